"""Which sizes mixed precision sends to the tensor cores does not depend on how the
ladder is cut into blocks."""
import numpy as np
import pytest

import ecgpu

pytestmark = pytest.mark.gpu


def _step(ctx, T1, T2, prec):
    ctx.set_precision(prec)
    try:
        ctx.cc_load(T1, T2)
        out = ctx.cc_step()
        return out, *ctx.cc_store()
    finally:
        ctx.set_precision(ecgpu.ECG_PREC_FP64)


@pytest.mark.parametrize("no,nv,nq,mixed", [
    # below 2^26 multiply-adds a product on an eighth of the virtual space: FP64
    (3, 20, 60, False), (6, 33, 140, False), (6, 40, 150, False),
    # from v * (v / 8) * v^2 * nQ = 2^26 on the V build runs on the tensor cores
    (4, 48, 120, True), (6, 64, 150, True), (4, 97, 160, True)])
def test_small_mixed_iterations_are_fp64(ctx, no, nv, nq, mixed):
    from ecgpu.synthetic import make_system
    B, h1, e0, _ = make_system(no, nv, nq, seed=8)
    ctx.set_system(B, h1, e0, no)
    _, T1, T2 = ctx.mp2()
    ref = _step(ctx, T1, T2, ecgpu.ECG_PREC_FP64)
    got = _step(ctx, T1, T2, ecgpu.ECG_PREC_MIXED)
    same = [np.array_equal(x, y) for x, y in zip(got, ref)]
    assert all(same) != mixed, same
    # three-slice products: 2^-23 of sums that average out, of amplitudes below 0.1
    assert np.abs(got[2] - ref[2]).max() < 1e-7
