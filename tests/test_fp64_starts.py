"""The FP64 operations on the integer pipe over every operand of the hardware
estimates that they start from: every leading mantissa (24 bits) at both
parities of the exponent, alone and with more bits below it, gives IEEE's
results. So no estimate lies outside the interval that the start's bits assume."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEADING = 1 << 23


def _check(mantissa, exponent, rng):
    """b = 1.mantissa 2^exponent (52 bits), a random."""
    from knc import abi
    n = len(mantissa)
    x = np.empty((n, 2))
    x[:, 0] = rng.uniform(1.0, 2.0, n)
    x[:, 1] = (mantissa + (np.int64(1023 + exponent) << 52)).view(np.float64)
    out = np.empty((n, 6))
    assert abi.load().knc_test_fp64_ops(abi.dptr(x), n, abi.dptr(out)) == 0
    a, b = x[:, 0], x[:, 1]
    w = np.sqrt(b)
    for col, want in enumerate((a / b, 1.0 / b, w, a / w)):
        assert np.array_equal(out[:, col], want), (col, b[out[:, col] != want][:3])


@pytest.mark.parametrize("low", ["none", "random"])
@pytest.mark.parametrize("exponent", [0, 1])
def test_every_leading_mantissa(exponent, low):
    rng = np.random.default_rng(3 + exponent)
    step = 1 << 20
    for first in range(0, LEADING, step):
        mantissa = np.arange(first, first + step, dtype=np.int64) << 29
        if low == "random":
            mantissa += rng.integers(0, 1 << 29, step)
        _check(mantissa, exponent, rng)


@pytest.mark.parametrize("exponent", [0, 1])
def test_next_to_powers_of_two(exponent):
    """The first and last leading mantissas at the ends and the middle of what
    FP32 rounds to one operand."""
    lead = np.concatenate([np.arange(0, 4096), np.arange(LEADING - 4096, LEADING)]).astype(np.int64)
    low = np.array([0, 1, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1], dtype=np.int64)
    _check(((lead[:, None] << 29) + low).reshape(-1), exponent, np.random.default_rng(7))
