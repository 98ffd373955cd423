"""Results of tens of megabytes reach fresh pageable arrays and pinned ones alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_amplitudes_to_pageable_and_pinned_memory(ctx):
    import torch
    from ecgpu.synthetic import make_system
    no, nv = 13, 161  # T2: 35 MB, 66 chunks and a remainder
    B, h1, e0, _ = make_system(no, nv, 40, seed=3)
    ctx.set_system(B, h1, e0, no)
    _, T1, T2 = ctx.mp2()
    pin = torch.zeros(no, no, nv, nv, dtype=torch.float64, pin_memory=True).numpy().T
    _, P2 = ctx.cc_store(np.zeros((nv, no), order="F"), pin)
    assert np.isfinite(T2).all() and np.abs(T2).max() > 0
    assert np.array_equal(T2, P2)
    for _ in range(3):
        assert np.array_equal(ctx.cc_store()[1], P2)
