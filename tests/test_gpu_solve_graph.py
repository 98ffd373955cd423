"""A solve, whose iterations from the third on are one recorded graph, gives the
bits of the same iterations made one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nv,nq,dc,mixed", [
    (1, 1, 3, False, False), (2, 3, 8, True, False), (5, 19, 60, False, False),
    (7, 40, 90, True, False), (6, 33, 80, False, True)])
def test_solve_equals_single_iterations(ctx, no, nv, nq, dc, mixed):
    import ecgpu
    from ecgpu.synthetic import make_system
    B, h1, e0, _ = make_system(no, nv, nq, seed=11)
    ctx.set_system(B, h1, e0, no)
    _, T1, T2 = ctx.mp2()
    opts = ctx.opts()
    opts.maxit = 12
    try:
        ctx.set_precision(ecgpu.ECG_PREC_MIXED if mixed else ecgpu.ECG_PREC_FP64)
        for _ in range(2):
            r = ctx.cc_solve(T1, T2, dc=dc, opts=opts)
        ctx.cc_load(T1, T2, opts=opts)
        for _ in range(r["iterations"]):
            out = ctx.cc_step(dc=dc)
            if mixed and out[3] < 100.0 * opts.thr:
                ctx.set_precision(ecgpu.ECG_PREC_FP64)
        S1, S2 = ctx.cc_store()
    finally:
        ctx.set_precision(ecgpu.ECG_PREC_FP64)
    assert r["iterations"] >= 3
    assert out[0] == r["E"] and out[3] == r["NormR"]
    assert np.array_equal(S1, r["T1"]) and np.array_equal(S2, r["T2"])
