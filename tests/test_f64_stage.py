"""The FP64 stage's integer-pipe arithmetic against IEEE results formed on the
host, and its update items at the edges of their columns and rows against the
oracle, bit for bit."""
import numpy as np
import pytest

from helpers import make_pair, zone_relative_errors

pytestmark = pytest.mark.gpu


def _pairs(kind):
    rng = np.random.default_rng(11)
    n = 400_000
    if kind == "random":
        x = rng.uniform(1.0, 2.0, (n, 2)) * np.exp2(rng.integers(-390, 390, (n, 2))) * rng.choice([-1.0, 1.0], (n, 2))
        x[::97, 0] = 0.0
        return x
    # quotients and roots next to midpoints: few-bit numbers moved by a few
    # units in the last place, and numbers just off powers of two
    if kind == "simple":
        a = rng.integers(1, 65, (n, 2)) * rng.choice([1.0, 0.1], (n, 2))
    else:
        a = np.exp2(rng.integers(-8, 9, (n, 2)))
    k = rng.integers(-8, 9, (n, 2)) if kind == "simple" else rng.integers(-(1 << 22), 1 << 22, (n, 2))
    return (a.view(np.int64) + k).view(np.float64)


@pytest.mark.parametrize("kind", ["random", "simple", "powers"])
def test_fp64_ops_round_like_ieee(kind):
    from knc import abi
    x = np.ascontiguousarray(_pairs(kind))
    out = np.empty((len(x), 6))
    assert abi.load().knc_test_fp64_ops(abi.dptr(x), len(x), abi.dptr(out)) == 0
    a, b = x[:, 0], x[:, 1]
    w = np.sqrt(np.abs(b))
    for col, want in enumerate((a / b, 1.0 / b, w, a / w, np.minimum(a, b), np.maximum(a, b))):
        assert np.array_equal(out[:, col], want), col


@pytest.mark.parametrize("order", ["RK1", "RK2", "RK3"])
@pytest.mark.parametrize("nr,nq", [(2, 16), (5, 31), (7, 33), (34, 64), (40, 97)])
@pytest.mark.parametrize("flow", ["wind", "jet", "sphere"])
def test_update_items_match_oracle(flow, nr, nq, order):
    """Items of 1 to 32 rows and partial columns; flows with supersonic and
    subsonic faces, HLLC and HLLE, through the fold and the host-state step."""
    from knc import workloads
    from knc.solver import PinnedArray
    w = {"wind": workloads.wind_small, "jet": workloads.jet_small, "sphere": workloads.sphere_small}[flow]()
    w.mesh.block_size = nr
    w.mesh.num_radial_zones = 82 if flow != "jet" else 400
    w.mesh.outer_radius = 1.6
    w.mesh.num_polar_zones = nq
    w.hydro.runge_kutta_order = order
    w.hydro.riemann_solver = "HLLC" if nr % 2 else "HLLE"
    for shape in (None, dict(tile_rows=4), dict(tile_rows=16), dict(tile_rows=64, strip=True)):
        g, o = make_pair(w)
        if shape:
            g.set_tuning(**shape)
        g.advance(2)
        o.advance(2)
        assert max(zone_relative_errors(g.state(), o.state())) == 0.0, shape
        assert g.time() == o.time()
    n = sum(a.shape[0] * a.shape[1] for a, _ in o.state().values())
    cons, scal = PinnedArray((n, 4)), PinnedArray((n,))
    cons.array[...] = np.concatenate([c.reshape(-1, 4) for _, (c, _) in sorted(o.state().items())])
    scal.array[...] = np.concatenate([s.reshape(-1) for _, (_, s) in sorted(o.state().items())])
    g.advance_host(cons.array, scal.array, 1)
    o.advance(1)
    assert np.array_equal(cons.array, np.concatenate([c.reshape(-1, 4) for _, (c, _) in sorted(o.state().items())]))
    assert np.array_equal(scal.array, np.concatenate([s.reshape(-1) for _, (_, s) in sorted(o.state().items())]))


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("order", ["RK2", "RK3"])
def test_host_state_chunks_on_a_larger_grid(precision, order):
    """Grids large enough to be split into chunks: the host-state step equals
    upload, advance and download."""
    import knc
    from knc import workloads
    from knc.solver import PinnedArray
    w = workloads.wind_small()
    w.mesh.block_size = 11
    w.mesh.num_radial_zones = 460
    w.mesh.outer_radius = 2.0
    w.mesh.num_polar_zones = 1010
    w.hydro.runge_kutta_order = order
    mode = knc.abi.KNC_PRECISION_MIXED if precision == "mixed" else knc.abi.KNC_PRECISION_FP64
    s = knc.build_solver(w, precision=mode)
    n = w.zones
    assert n >= 4 * 65536
    ci, si, co, so = (PinnedArray(k) for k in ((n, 4), (n,), (n, 4), (n,)))
    s.get_state(ci.array, si.array)
    s.advance_host(ci.array, si.array, 1, co.array, so.array)
    want_c, want_s = np.empty((n, 4)), np.empty(n)
    s.set_state(ci.array, si.array)
    s.advance(1)
    s.get_state(want_c, want_s)
    assert np.array_equal(co.array, want_c) and np.array_equal(so.array, want_s)
    assert not np.array_equal(co.array, ci.array)


@pytest.mark.parametrize("nr,nq,zones", [(5, 40, 90), (13, 97, 210), (40, 240, 330), (64, 700, 500)])
def test_mixed_strips_and_recovery_runs(nr, nq, zones):
    """Strips and recovery runs of one to many rows, with and without columns
    that fill a CTA (97 and 700 zones: 4 and 22 columns of 32; 240: 8): the bits
    of the tile form."""
    import knc
    from knc import workloads
    w = workloads.jet_small()
    w.mesh.block_size = nr
    w.mesh.num_radial_zones = zones
    w.mesh.num_polar_zones = nq
    states = []
    for t in (dict(tile_rows=8), dict(tile_rows=16, strip=True, deferred=True)):
        g = knc.build_solver(w)
        g.set_precision(knc.abi.KNC_PRECISION_MIXED)
        g.set_tuning(**t)
        g.advance(4)
        states.append(g.state())
    assert max(zone_relative_errors(states[1], states[0])) == 0.0
