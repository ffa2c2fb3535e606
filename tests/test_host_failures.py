"""A failing host-state step whose chunks run side by side: one chunk's failure
appears while the kernels of the others start. Whatever they do then, the
recovery's statistics count whole zones, the failure is the poisoned zone's,
and a state set afterwards advances as in a new solver."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("guess", ["plain", "learned"])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("order", ["RK2", "RK3"])
def test_failure_beside_other_chunks(order, precision, guess, trained_mlp):
    import knc
    from knc import workloads
    from knc.solver import PinnedArray
    w = workloads.wind_small()
    w.mesh.block_size = 11
    w.mesh.num_radial_zones = 460
    w.mesh.outer_radius = 2.0
    w.mesh.num_polar_zones = 1010
    w.hydro.runge_kutta_order = order
    solvers = []
    for _ in range(2):
        s = knc.build_solver(w, precision=knc.abi.KNC_PRECISION_MIXED if precision == "mixed"
                             else knc.abi.KNC_PRECISION_FP64)
        if guess == "learned":
            s.set_c2p_guess(knc.abi.KNC_GUESS_MLP, trained_mlp[0])
        solvers.append(s)
    s, fresh = solvers
    n, nq, stages = w.zones, 1010, int(order[2])
    good_c, good_s = np.empty((n, 4)), np.empty(n)
    s.get_state(good_c, good_s)
    cons, scal, cons_out, scal_out = (PinnedArray(k) for k in ((n, 4), (n,), (n, 4), (n,)))
    scal.array[...] = good_s
    # at most: every zone and the rows beside the (at most 10) chunks' ends, each stage
    most = stages * (n + 9 * 2 * 2 * stages * nq)
    for k in range(12):
        s.init_from_model(0.0)   # (a failed solver asks for a state first)
        cons.array[...] = good_c
        block, zone = 1 + 2 * k, 5 * nq + 77 * k
        cons.array[block * 11 * nq + zone, 0] = -1.0
        s.reset_c2p_stats()
        with pytest.raises(knc.HydroError) as exc:
            s.advance_host(cons.array, scal.array, 1, cons_out.array, scal_out.array)
        e = exc.value.error
        assert (e["kind"], e["block"], e["i"], e["j"]) == ("NegativeDensity", block, zone // nq, zone % nq)
        st = s.c2p_stats()
        assert 0 < st["zones"] <= most
        assert st["iters_fp64"] <= 200 * st["zones"] and st["iters_fp32"] <= 64 * st["zones"]
        assert st["fallbacks"] <= st["zones"]
    for x in (s, fresh):
        x.init_from_model(0.0)
        cons.array[...] = good_c
        x.advance_host(cons.array, scal.array, 1, cons_out.array, scal_out.array)
    a, b = s.state(), fresh.state()
    assert all(np.array_equal(x, y) for i in a for x, y in zip(a[i], b[i]))
