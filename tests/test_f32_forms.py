"""The mixed stage's one-instruction reciprocals and roots: the plain forms'
bits on every mantissa, and a flow whose wave speeds differ by less than FP32's
smallest normal number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-126, -125, -61, -2, -1, 0, 1, 2, 60, 124, 125])
def test_forms_have_the_plain_bits(exponent):
    """(2^126 and above: the reciprocal's result is subnormal and flushed)"""
    from knc import abi
    rng = np.random.default_rng(exponent + 200)
    n = 1 << 23
    x = np.empty((n, 2), dtype=np.float32)
    x[:, 1] = (np.arange(n, dtype=np.int32) + ((127 + exponent) << 23)).view(np.float32)
    # (quotients inside the normal range)
    x[:, 0] = rng.uniform(1.0, 2.0, n) * np.exp2(np.clip(exponent, -60, 60)) * rng.choice([-1.0, 1.0], n)
    out = np.empty((n, 8), dtype=np.float32)
    assert abi.load().knc_test_f32_forms(abi.fptr(x), n, abi.fptr(out)) == 0
    for k in range(4):
        assert np.array_equal(out[:, 2 * k].view(np.int32), out[:, 2 * k + 1].view(np.int32)), k


@pytest.mark.parametrize("tuning", [dict(tile_rows=8), dict(tile_rows=16, strip=True, deferred=True)])
def test_gas_without_pressure_at_the_smallest_speeds(tuning):
    """Zones without pressure that part at 4e-39 of the speed of light: nothing
    moves, and every flux is a number."""
    import knc
    from knc import workloads
    w = workloads.wind_small()
    w.mesh.num_polar_zones = 32
    g = knc.build_solver(w)
    g.set_precision(knc.abi.KNC_PRECISION_MIXED)
    g.set_tuning(**tuning)
    rng = np.random.default_rng(5)
    before = {}
    for k in g.block_indexes():
        cons, scal = g.get_block(k)
        mass = 1e10 * cons[..., 0]
        cons = np.stack([mass, *(4e-39 * mass * rng.choice([-1.0, 1.0], (2, *mass.shape))), 0.0 * mass], axis=-1)
        g.add_block(k, cons, scal)
        before[k] = cons
    g.advance(1)
    inner = g.block_indexes()[1:-1]   # (the wind of the model enters the first and borders the last)
    for k in inner:
        cons, scal = g.get_block(k)
        assert np.all(np.isfinite(cons)) and np.all(np.isfinite(scal))
        assert np.array_equal(cons[..., 0], before[k][..., 0]) and np.all(cons[..., 3] == 0.0)
