"""Mixed (T) with more occupied pairs than the operand split takes in one go."""
import numpy as np
import pytest

import ecgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no,nv,nq", [(22, 5, 30), (23, 6, 30), (33, 5, 40)])  # 484, 529, 1089 pairs
def test_mixed_pert_t_matches_fp64(ctx, no, nv, nq):
    from ecgpu.synthetic import make_system
    B, h1, e0, _ = make_system(no, nv, nq, seed=7)
    ctx.set_system(B, h1, e0, no)
    _, T1, T2 = ctx.mp2()
    T1 = 0.02 * np.random.default_rng(nv).standard_normal((nv, no))
    ref = ctx.pert_t(T1, T2)
    ctx.set_precision(ecgpu.ECG_PREC_MIXED)
    try:
        got = ctx.pert_t(T1, T2)
    finally:
        ctx.set_precision(ecgpu.ECG_PREC_FP64)
    # two-slice products, 2^-16 of each term, averaging over the triplets' v^3 of them
    for x, y in zip(got, ref):
        assert abs(x - y) < 2e-5 * abs(y)
