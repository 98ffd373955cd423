"""Bounded device-side waits that run out (a 1 ns bound, ECG_OPT_TC_WAIT_NS: the
kernels record it, let their own copies land and return): the call that ran them
reports ECG_ERR_TIMEOUT, no other call does, and the context stays usable."""
import threading

import numpy as np
import pytest

import ecgpu
from ecgpu._lib import ECG_ERR_TIMEOUT, ECG_OPT_TC_WAIT_NS

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
