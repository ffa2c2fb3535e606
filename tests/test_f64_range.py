"""The FP64 stage at the ends of the number range: flows around the speed of
sound whose pressures run from 1e-300 to 1e280 (beyond what the FP32 estimate of
the supersonic faces can hold) against the oracle, and pressures that are no
number against the fused stage, whose faces all take the full solve, bit for
bit."""
import math

import numpy as np
import pytest

from helpers import make_pair

pytestmark = pytest.mark.gpu

NR, NQ = 8, 24
GAMMA = {"relativistic": 4.0 / 3.0, "newtonian": 5.0 / 3.0}
# decades of the blocks' pressures, close together where FP32 ends
DECADES = sorted([*range(-300, 281, 58), *range(-47, -28, 2), *range(29, 48, 2), 0])


def _workload(system, riemann):
    from knc import workloads
    w = workloads.wind_small() if system == "relativistic" else workloads.sphere_small()
    n = len(DECADES)
    w.mesh.block_size, w.mesh.num_polar_zones = NR, NQ
    w.mesh.num_radial_zones = round(NR / (10.0 ** (1.0 / n) - 1.0))
    w.mesh.outer_radius = (1.0 + NR / w.mesh.num_radial_zones) ** n * (1.0 - 1e-6)
    w.hydro.riemann_solver = riemann
    w.hydro.runge_kutta_order = "RK1"
    assert w.num_blocks == n
    return w


def _block(system, index, volume, temperature, decade, rng):
    """Conserved state of a block: p about 10^decade, p / rho about `temperature`,
    velocities up to twice the speed of sound, either way along either axis."""
    g = GAMMA[system]
    # densities whose squares (relativistic recovery) or selves stay in range
    most, shift = 140 if system == "relativistic" else 280, math.log10(temperature)
    decade = min(max(decade, shift - most), shift + most)
    p = 10.0 ** decade * (1.0 + rng.random((NR, NQ)))
    rho = p / temperature / (1.0 + rng.random((NR, NQ)))
    cs = np.sqrt(g * temperature / (1.0 + 4.0 * temperature if system == "relativistic" else 1.0))
    ur, uq = (cs * rng.uniform(-2.0, 2.0, (2, NR, NQ)))
    uu = ur * ur + uq * uq
    if system == "newtonian":
        u = [rho, rho * ur, rho * uq, p / (g - 1.0) + 0.5 * rho * uu]
    else:
        w = np.sqrt(1.0 + uu)
        d, gh = rho * w, g / (g - 1.0)
        m = d * (1.0 + gh * p / rho)
        u = [d, m * ur, m * uq, p * (gh * (1.0 + uu) - 1.0) + d * uu / (w + 1.0)]
    return np.stack([x * volume for x in u], axis=-1), 0.3 * u[0] * volume


def _advance_both(system, riemann, temperature, change=None):
    import knc_oracle
    w = _workload(system, riemann)
    g, o = make_pair(w)
    if change:
        o, _ = make_pair(w)
        o.set_tuning(tile_rows=8, fused=True)
    rng = np.random.default_rng(17)
    for k in o.block_indexes():
        volume = knc_oracle.block_geometry(w.mesh.to_c(), k)["dv"].reshape(NR, NQ)
        cons, scal = _block(system, k, volume, temperature, DECADES[k], rng)
        if change:
            change(k, cons)
        for s in (g, o):
            s.add_block(k, cons, scal)
    speed = math.sqrt(temperature) * (3e10 if system == "relativistic" else 1.0)
    dt = 0.1 / w.mesh.num_radial_zones / min(speed, 3e10 if system == "relativistic" else speed)
    g.advance(1, dt)
    o.advance(1, dt)
    return g.state(), o.state()


def _assert_same(a, b):
    for k in sorted(b):
        for x, y in zip(a[k], b[k]):
            assert np.array_equal(x, y, equal_nan=True), (k, DECADES[k])


@pytest.mark.parametrize("temperature", [1e-45, 1e-40, 1e-20, 1e-11, 1e-7, 1e-2])
@pytest.mark.parametrize("riemann", ["HLLE", "HLLC"])
@pytest.mark.parametrize("system", ["relativistic", "newtonian"])
def test_faces_at_the_ends_of_the_range(system, riemann, temperature):
    _assert_same(*_advance_both(system, riemann, temperature))


@pytest.mark.parametrize("riemann", ["HLLE", "HLLC"])
@pytest.mark.parametrize("temperature", [1e10, 1e30])
def test_hot_newtonian_faces(riemann, temperature):
    _assert_same(*_advance_both("newtonian", riemann, temperature))


@pytest.mark.parametrize("riemann", ["HLLE", "HLLC"])
@pytest.mark.parametrize("temperature", [1e-7, 1e-10, 1e-39])
@pytest.mark.parametrize("value", [math.nan, math.inf])
def test_pressures_that_are_no_number(riemann, temperature, value):
    """A zone in seven without a pressure beside supersonic neighbours; at some
    of the densities FP32's largest number over them is still below the square of
    these velocities. Which of a wave speed and no number is the lesser differs between
    C++'s std::min and the device's form, so the other side here is the device's
    own plain solve."""
    def change(k, cons):
        cons[..., 1] = 4e12 * cons[..., 0]
        cons[..., 2] = 3e12 * cons[..., 0]
        cons[..., 3] += 12.5e24 * cons[..., 0]
        cons.reshape(-1, 4)[k % 7::7, 3] = value
    _assert_same(*_advance_both("newtonian", riemann, temperature, change))
