"""FP64 products and the particle ladder at odd sizes: operands that TMA cannot
address as they lie, a-blocks of V that start inside the virtual space."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("tb", ["N", "T"])
@pytest.mark.parametrize("m,n,k", [(301, 277, 1031), (65, 1023, 513), (640, 642, 643),
                                   (33, 31, 2047), (1, 127, 129), (129, 1, 4097)])
def test_odd_gemm_matches_numpy(ctx, ta, tb, m, n, k):
    """Odd pitches, with one or both operands copied into even ones or neither."""
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((k, m) if ta == "T" else (m, k))
    B = rng.standard_normal((n, k) if tb == "T" else (k, n))
    C0 = rng.standard_normal((m, n))
    out = ctx.diag_gemm(ta, tb, 0.7, A, B, -1.3, C0)
    opA, opB = (A.T if ta == "T" else A), (B.T if tb == "T" else B)
    ref = 0.7 * (opA @ opB) - 1.3 * C0
    bound = (k + 8) * 2.0 ** -53 * (np.abs(opA) @ np.abs(opB) + 1.3 * np.abs(C0))
    assert (np.abs(out - ref) <= 2.0 * bound).all()


@pytest.mark.parametrize("no,nv,nq", [(2, 81, 21), (3, 96, 20), (2, 107, 18)])
def test_residual_over_several_ladder_blocks(ctx, no, nv, nq):
    from ecgpu.synthetic import make_system
    from oracle.dfcc import DFCC
    B, h1, e0, _ = make_system(no, nv, nq, seed=5)
    d = DFCC(B, h1, e0, no)
    d.start()
    rng = np.random.default_rng(nv)
    d.T1 = 0.02 * rng.standard_normal((nv, no))
    for name, _, fn in d.iteration_tasks():
        if name.startswith("update"):
            break
        fn()
    ctx.set_system(B, h1, e0, no)
    R1, R2 = ctx.cc_residual(d.T1, np.asfortranarray(d.T2))
    assert np.abs(R1 - d.R1).max() < 1e-12 and np.abs(R2 - d.R2).max() < 1e-12
