"""FP64 (T) on the TMA-staged K builds: repeatable to the bit, and equal to the
density-fitted numpy restatement."""
import numpy as np
import pytest

from ecgpu._lib import ECG_OPT_TRIPLES_BATCH

pytestmark = pytest.mark.gpu


def _system(no, nv, nq, seed=7):
    from ecgpu.synthetic import make_system
    B, h1, e0, _ = make_system(no, nv, nq, seed=seed)
    return B, h1, e0


def test_pert_t_repeats_to_the_bit(ctx):
    """Every pass gives the same bits, whatever the batches: the K builds add
    in a fixed order, so a difference is a stage that was refilled while a
    warp still had to read it (seen at this size before the release was moved
    behind the MMAs: one pass in ten)."""
    B, h1, e0 = _system(3, 150, 200)
    ctx.set_system(B, h1, e0, 3)
    ctx.mp2()
    first = ctx.pert_t()
    try:
        for nb in (0, 1, 3):
            ctx.set_option(ECG_OPT_TRIPLES_BATCH, nb)
            for _ in range(12):
                assert ctx.pert_t() == first
    finally:
        ctx.set_option(ECG_OPT_TRIPLES_BATCH, 0)


@pytest.mark.parametrize("no,nv,nq", [(2, 10, 30), (3, 19, 60), (4, 33, 90), (3, 48, 100),
                                      (3, 65, 120), (5, 80, 130), (3, 97, 150), (2, 130, 170)])
def test_pert_t_matches_restatement(ctx, no, nv, nq):
    """Odd and even virtual counts around the tile edges."""
    from oracle.dfcc import DFCC
    B, h1, e0 = _system(no, nv, nq)
    d = DFCC(B, h1, e0, no)
    d.start()
    rng = np.random.default_rng(no + nv)
    T1 = 0.02 * rng.standard_normal((nv, no))
    ref = d.pert_t(T1, d.T2)
    ctx.set_system(B, h1, e0, no)
    got = ctx.pert_t(T1, np.asfortranarray(d.T2))
    # sums of ~nv^3 terms of either sign: 1e-12 of the energy's size
    assert abs(got[0] - ref[0]) < 1e-12 and abs(got[1] - ref[1]) < 1e-12


@pytest.mark.parametrize("no,nv,nq", [(2, 9, 30), (4, 33, 60), (3, 64, 80), (3, 129, 90),
                                      (7, 100, 110), (2, 257, 60), (2, 300, 60)])
def test_mixed_pert_t_matches_fp64(ctx, no, nv, nq):
    """Tensor-core tile widths at their edges (one tile of 16 to 256 columns, two
    beyond), chunks of triplets that are full and not."""
    import ecgpu
    B, h1, e0 = _system(no, nv, nq)
    ctx.set_system(B, h1, e0, no)
    _, T1, T2 = ctx.mp2()
    T1 = 0.02 * np.random.default_rng(nv).standard_normal((nv, no))
    ref = ctx.pert_t(T1, T2)
    ctx.set_precision(ecgpu.ECG_PREC_MIXED)
    try:
        got = ctx.pert_t(T1, T2)
        assert ctx.pert_t(T1, T2) == got
    finally:
        ctx.set_precision(ecgpu.ECG_PREC_FP64)
    # two-slice products, 2^-16 of each term, averaging over v^3 of them
    for x, y in zip(got, ref):
        assert abs(x - y) < 2e-5 * abs(y)
