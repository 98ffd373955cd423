"""Bounded device-side waits that run out (a 1 ns bound, ECG_OPT_TC_WAIT_NS: the
kernels record it, let their own copies land and return): the call that ran them
reports ECG_ERR_TIMEOUT, no other call does, and the context stays usable."""
import threading

import numpy as np
import pytest

import ecgpu
from ecgpu._lib import ECG_ERR_OOM, ECG_ERR_TIMEOUT, ECG_OPT_TC_WAIT_NS

pytestmark = pytest.mark.gpu


def test_time_outs_stay_with_their_context():
    """Two contexts on two host threads, one whose every wait runs out: it reports
    each of its time-outs, the other none."""
    rng = np.random.default_rng(2)
    m, n, k = 256, 192, 4096
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    ref = A @ B
    gate = threading.Barrier(2)
    seen, wrong = [], []

    def short():
        with ecgpu.Context(0) as c:
            c.set_option(ECG_OPT_TC_WAIT_NS, 1)
            gate.wait()
            for _ in range(60):
                try:
                    c.diag_gemm("N", "N", 1.0, A, B, 0.0, np.zeros((m, n)))
                    seen.append(0)
                except ecgpu.ECGError as e:
                    seen.append(e.code)

    def plain():
        with ecgpu.Context(0) as c:
            gate.wait()
            for _ in range(60):
                try:
                    out = c.diag_gemm("N", "N", 1.0, A, B, 0.0, np.zeros((m, n)))
                    if not np.abs(out - ref).max() < 1e-10:
                        wrong.append("result")
                except ecgpu.ECGError as e:
                    wrong.append(e.code)

    threads = [threading.Thread(target=f) for f in (short, plain)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == [ECG_ERR_TIMEOUT] * 60
    assert not wrong, wrong


def _calls(mixed):
    """(name, kernels, call) of the entry points that queue kernels with bounded waits, on
    a system that is set; `kernels`: codes of which one has to be reported."""
    from ecgpu.basis import ShellArrays
    from ecgpu.synthetic import make_system
    no, nv, nq = 4, 36, 96
    B, h1, e0, _ = make_system(no, nv, nq, seed=9)
    rng = np.random.default_rng(1)
    with ecgpu.Context(0) as c:
        c.set_system(B, h1, e0, no)
        _, T1, T2 = c.mp2()
    T1 = np.asfortranarray(0.02 * rng.standard_normal((nv, no)))
    U1, U2 = 2.0 * T1, 2.0 * T2 - T2.transpose(1, 0, 2, 3)
    # 28 functions: an even pitch, which the kernels with waits can read
    ao = ShellArrays([0, 1, 2] * 3 + [0], [2, 1, 1] * 3 + [1], rng.uniform(-1, 1, 30),
                     rng.uniform(0.3, 2.0, 13), np.ones(13), [0, 1, 2] * 3 + [0])
    M = np.asfortranarray(rng.standard_normal((ao.nbf, ao.nbf - 1)))
    C = np.asfortranarray(rng.standard_normal((ao.nbf, ao.nbf - 3)))
    gemm, kb = {17}, {65, 66, 67, 68} if mixed else {49}

    def df(call):
        def run(c):
            c.set_option(ECG_OPT_TC_WAIT_NS, 0)
            with c.df_factors(ao, ao, M) as d:
                c.set_option(ECG_OPT_TC_WAIT_NS, c.bound)
                return call(d)
        return run

    def step(c):
        c.cc_load(T1, T2)
        c.cc_step()
        return c.cc_store()

    def step_host(c):
        c.cc_load(T1, T2)
        X1, X2 = T1.copy(order="F"), T2.copy(order="F")
        return c.cc_step_host(X1, X2), X1, X2

    def solve(c):
        r = c.cc_solve(T1, T2, opts=c.opts(maxit=4))
        return r["T1"], r["T2"]

    def lam(c):
        return c.lambda_solve(T1, T2, opts=c.opts(maxit=3))["U2"]

    def system(c):
        c.set_system(B, h1, e0, no)
        return c.mp2()[2]

    return [
        ("cc_residual", gemm, lambda c: c.cc_residual(T1, T2)),
        ("cc_step", gemm, step),
        ("cc_step_host", gemm, step_host),
        ("cc_solve", gemm, solve),
        ("pert_t", kb, lambda c: c.pert_t(T1, T2)),
        ("lambda_pert_t", kb, lambda c: c.lambda_pert_t(T1, T2, U1, U2)),
        ("lambda_residual", gemm, lambda c: c.lambda_residual(T1, T2, U1, U2)),
        ("lambda_solve", gemm, lam),
        ("one_rdm", gemm, lambda c: c.one_rdm(T1, T2, U1, U2)),
        ("energy_gradient", gemm, lambda c: c.energy_gradient(T1, T2, U1, U2)),
        ("df_create", gemm, lambda c: c.df_factors(ao, ao, M).close()),
        ("df_fock", gemm, df(lambda d: d.fock(np.eye(ao.nbf), C[:, :4]))),
        ("df_mo", gemm, df(lambda d: d.mo(C))),
        ("set_system", gemm, system),
    ]


def _flat(x):
    if x is None:
        return []
    if isinstance(x, (tuple, list)):
        return [z for y in x for z in _flat(y)]
    return [np.asarray(x)]


@pytest.mark.parametrize("mixed", [False, True])
def test_every_call_reports_its_time_outs(mixed):
    """With every wait running out each call that rests on such kernels reports it, and
    names the kernels; afterwards it gives the bits it gave before."""
    calls = _calls(mixed)
    with ecgpu.Context(0) as c:
        if mixed:
            c.set_precision(ecgpu.ECG_PREC_MIXED)
        c.bound = 0
        calls[-1][2](c)  # the system
        before = [_flat(call(c)) for _, _, call in calls]
        for (name, kernels, call), ref in zip(calls, before):
            c.bound = 1
            c.set_option(ECG_OPT_TC_WAIT_NS, 1)
            try:
                call(c)
                raised = None
            except ecgpu.ECGError as e:
                raised = e
            finally:
                c.bound = 0
                c.set_option(ECG_OPT_TC_WAIT_NS, 0)
            assert raised is not None and raised.code == ECG_ERR_TIMEOUT, (name, raised)
            codes = {int(x) for x in str(raised).split("code ")[1].split(")")[0].split(",")}
            assert codes & kernels, (name, codes)
            got = _flat(call(c))
            assert len(got) == len(ref) and all(np.array_equal(x, y) for x, y in zip(got, ref)), name


def test_a_call_that_fails_leaves_no_time_out_behind():
    """A (T) call that the memory cap stops behind GEMMs whose waits ran out reports
    the cap, and the calls after it do not report the time-outs."""
    from ecgpu.synthetic import make_system
    B, h1, e0, _ = make_system(3, 30, 64, seed=4)
    with ecgpu.Context(0) as c:
        c.set_system(B, h1, e0, 3)
        e_mp2, T1, T2 = c.mp2()
        cap = 0
        while True:
            cap += 1 << 17
            c.set_mem_cap(cap)
            c.set_option(ECG_OPT_TC_WAIT_NS, 1)
            with pytest.raises(ecgpu.ECGError) as e:
                c.pert_t()
            c.set_option(ECG_OPT_TC_WAIT_NS, 0)
            assert e.value.code == ECG_ERR_OOM, e.value
            if "vvvo slab" in str(e.value):
                break
        assert c.mp2()[0] == e_mp2
