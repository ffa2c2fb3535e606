"""The launch shape of a solver nobody tuned: giving a solver the tuning it
reports changes nothing, and the autotuner offers that shape too."""
import pytest

pytestmark = pytest.mark.gpu


def _update_ms(s):
    """Update kernels of 10 steps, the fastest of three runs."""
    best = []
    for _ in range(3):
        s.set_profiling(False)
        s.set_profiling(True)
        before = s.kernel_times()["update"][0]
        s.advance(10)
        best.append(s.kernel_times()["update"][0] - before)
    s.set_profiling(False)
    return min(best)


def test_reported_tuning_is_neutral_and_a_candidate():
    """256 x 128 FP64 wind, whose grid-chosen tiles run in half the time of
    items of 8 rows: the margins here lie far from both."""
    import knc
    from knc import workloads
    w = workloads.wind_small()
    default, given, tuned = (knc.build_solver(w) for _ in range(3))
    for s in (default, given, tuned):
        s.advance(2)
    want = _update_ms(default)
    t = given.tuning()
    given.set_tuning(**t)
    assert given.tuning() == t
    assert _update_ms(given) < 1.4 * want
    given.set_tuning(tile_rows=16)
    assert _update_ms(given) > 2.0 * want     # (another shape is another shape)
    given.set_tuning(**t)
    assert _update_ms(given) < 1.4 * want     # and there is a way back
    tuned.autotune(reps=3)
    if not tuned.tuning()["fused"]:
        assert _update_ms(tuned) < 1.4 * want
