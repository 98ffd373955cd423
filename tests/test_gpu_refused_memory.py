"""Calls that the memory cap stops half way: a status, no pointer to memory that is
not there, and a context that goes on."""
import numpy as np
import pytest

import ecgpu
from ecgpu._lib import ECG_ERR_OOM, ECG_ERR_STATE

pytestmark = pytest.mark.gpu


def _system(no, nv, nq):
    from ecgpu.synthetic import make_system
    B, h1, e0, _ = make_system(no, nv, nq, seed=6)
    return B, h1, e0, no


def _close(x, y):
    """Equal but for the order of sums: where memory is short, products of odd pitch run
    on the kernel that splits K elsewhere.  At most 1e5 terms, of amplitudes and
    integrals whose products add up to less than 1: 1e5 * 2^-53, some of it averaging."""
    return all(np.abs(a - b).max() < 1e-13 * max(1.0, np.abs(b).max()) for a, b in zip(x, y))


def test_lambda_residual_under_a_growing_cap():
    """Refused at each of its buffers and at the larger workspace in turn; after each
    refusal the residual still runs, and the first call that fits is right."""
    with ecgpu.Context(0) as c:
        c.set_system(*_system(3, 20, 40))
        _, T1, T2 = c.mp2()
        U1, U2 = 2.0 * T1, 2.0 * T2 - T2.transpose(1, 0, 2, 3)
        ref = c.cc_residual(T1, T2)
        refused, cap = set(), 0
        while True:
            cap += 1 << 14
            c.set_mem_cap(cap)
            try:
                R = c.lambda_residual(T1, T2, U1, U2)
                break
            except ecgpu.ECGError as e:
                assert e.code == ECG_ERR_OOM
                refused.add(str(e).rsplit(" ", 1)[1])
            assert _close(c.cc_residual(T1, T2), ref)
        assert {"U", "RU", "workspace"} <= refused, refused
        c.set_mem_cap(0)
        with ecgpu.Context(0) as d:
            d.set_system(*_system(3, 20, 40))
            assert _close(R, d.lambda_residual(T1, T2, U1, U2))


def test_iterations_without_their_history():
    """A cc_load whose longer DIIS history is refused leaves none: a step then is a
    call-order error, and the next cc_load works."""
    with ecgpu.Context(0) as c:
        c.set_system(*_system(4, 24, 48))
        _, T1, T2 = c.mp2()
        c.cc_load(T1, T2, opts=c.opts(maxdiis=3))
        ref = c.cc_step()
        c.set_mem_cap(1 << 16)
        with pytest.raises(ecgpu.ECGError) as e:
            c.cc_load(T1, T2, opts=c.opts(maxdiis=6))
        assert e.value.code == ECG_ERR_OOM
        c.set_mem_cap(0)
        with pytest.raises(ecgpu.ECGError) as e:
            c.cc_step()
        assert e.value.code == ECG_ERR_STATE
        c.cc_load(T1, T2, opts=c.opts(maxdiis=6))
        assert np.array_equal(c.cc_step(), ref)


# bytes that a system took with blocks of an eighth of the virtual space in the
# ladder and term-by-term rings: set up, and with the Lambda equations' buffers
SIZES = [((5, 19, 60), 4654816, 11344880), ((12, 57, 200), 172595432, 186068024),
         ((16, 76, 280), 498504128, 569683648), ((1, 40, 60), 15056944, 15110400),
         ((20, 20, 60), 38081360, 43315280)]


@pytest.mark.parametrize("size,cap,cap_lambda", SIZES)
def test_systems_fit_the_memory_they_took(size, cap, cap_lambda):
    no, nv, nq = size
    sys_ = _system(no, nv, nq)
    with ecgpu.Context(0) as c, ecgpu.Context(0) as free:
        c.set_mem_cap(cap)
        for x in (c, free):
            x.set_system(*sys_)
        _, T1, T2 = c.mp2()
        T1 = 0.02 * np.random.default_rng(1).standard_normal(T1.shape)
        assert _close(c.cc_residual(T1, T2), free.cc_residual(T1, T2))
        c.set_mem_cap(cap_lambda)
        U1, U2 = 2.0 * T1, 2.0 * T2 - T2.transpose(1, 0, 2, 3)
        assert _close(c.lambda_residual(T1, T2, U1, U2), free.lambda_residual(T1, T2, U1, U2))


# a system and what (T) took beside it
SIZES_T = [((5, 19, 60), 4654816 + 2306000), ((10, 61, 200), 168437712 + 418787680),
           ((16, 76, 280), 498504128 + 1014903376), ((20, 20, 60), 38081360 + 21566328),
           ((17, 83, 304), 671143536 + 1330940256)]


@pytest.mark.parametrize("size,cap", SIZES_T)
def test_pert_t_fits_the_memory_it_took(size, cap):
    """At odd virtual counts the copies in even pitches come on top, which batches of
    fewer triplets make up for; the energies do not depend on the batches."""
    no, nv, nq = size
    sys_ = _system(no, nv, nq)
    with ecgpu.Context(0) as c, ecgpu.Context(0) as free:
        c.set_mem_cap(cap)
        for x in (c, free):
            x.set_system(*sys_)
            x.mp2()
        assert c.pert_t() == free.pert_t()


def test_copies_for_odd_pitches_keep_to_the_cap():
    """At an odd virtual count the FP64 GEMM copies operands into even pitches (0.2 GB
    here) where memory allows: not beyond a cap, and an allocation that needs the room
    gets it."""
    import torch
    size, cap, cap_lambda = (4, 181, 600), 4668903184, 5610650208
    sys_ = _system(*size)
    torch.cuda.mem_get_info()
    with ecgpu.Context(0) as c:
        c.set_mem_cap(cap)
        c.set_system(*sys_)
        _, T1, T2 = c.mp2()
        before = torch.cuda.mem_get_info()[0]
        ref = c.cc_residual(T1, T2)
        # 32 MiB of split-K partial products beside it
        assert before - torch.cuda.mem_get_info()[0] < 64 << 20
        c.set_mem_cap(0)
        got = c.cc_residual(T1, T2)
        assert before - torch.cuda.mem_get_info()[0] > 150 << 20
        assert _close(got, ref)
        c.set_mem_cap(cap_lambda)
        c.lambda_residual(T1, T2, 2.0 * T1, 2.0 * T2 - T2.transpose(1, 0, 2, 3))
        assert before - torch.cuda.mem_get_info()[0] < cap_lambda - cap + (64 << 20)


def test_workspace_is_free_after_a_refusal():
    """Mixed iterations that the cap stops inside the ladder (the storage of its BF16
    slices), again and again: the workspace they had taken is there for the next call."""
    size = (6, 64, 160)
    with ecgpu.Context(0) as c:
        c.set_system(*_system(*size))
        _, T1, T2 = c.mp2()
        ref = c.cc_residual(T1, T2)
        c.cc_load(T1, T2)
        c.set_precision(ecgpu.ECG_PREC_MIXED)
        c.set_mem_cap(1 << 16)
        for _ in range(4):
            with pytest.raises(ecgpu.ECGError) as e:
                c.cc_step()
            assert e.value.code == ECG_ERR_OOM and "split-operand" in str(e.value)
        c.set_mem_cap(0)
        c.set_precision(ecgpu.ECG_PREC_FP64)
        assert _close(c.cc_residual(T1, T2), ref)
