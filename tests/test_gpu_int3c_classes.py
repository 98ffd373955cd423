"""Every class (la >= lb) of the three-centre integral kernel against the
Obara-Saika oracle, with contracted shells (whose primitive pairs eight lanes
share) and single primitives, on fitting shells of all degrees."""
import numpy as np
import pytest

from oracle import ints as I
from test_gpu_ints import _oracle, _shells

pytestmark = pytest.mark.gpu

FIT = [(0, 1), (1, 2), (2, 1), (3, 1), (4, 1)]


@pytest.mark.parametrize("la,lb", [(a, b) for a in range(5) for b in range(a + 1)])
@pytest.mark.parametrize("prims", [(3, 2), (1, 1)])
def test_class_matches_oracle(ctx, la, lb, prims):
    """Both orders of a pair are the same bits, and a repeated call gives them again:
    each integral has one writer, pairs of a shell with itself among them."""
    ao, _ = _shells([(la, prims[0]), (lb, prims[1])], 40 + 5 * la + lb)
    fit, _ = _shells(FIT, 41)
    B = ctx.int3c2e(ao, fit)
    Bo = I.int3c2e(_oracle(ao), _oracle(fit))
    # sums of up to nine primitive pairs in FP64; the oracle's recursion is the looser side
    assert np.abs(B - Bo).max() < 1e-10 * np.abs(Bo).max()
    assert np.array_equal(B, B.transpose(1, 0, 2))
    for _ in range(3):
        assert np.array_equal(ctx.int3c2e(ao, fit), B)
