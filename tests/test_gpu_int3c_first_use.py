"""The first three-centre integrals of a process, asked for by several contexts at
once: the tables of the Boys functions that they share are complete before any of
them reads it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys, threading
sys.path[:0] = [{root!r}, {pkg!r}]
import numpy as np
import ecgpu
from ecgpu.basis import ShellArrays

ao = ShellArrays([0, 1, 2, 3], [2, 1, 1, 1], [0., 0., 0., 1., 0., 0., 0., 1.1, 0., .4, .3, 1.2],
                 [3., .6, .9, 1.1, .8], [.4, .7, 1., 1., 1.], [0, 1, 2, 3])
fit = ShellArrays([0, 2, 4], [1, 1, 1], [0., 0., 0., 1., 0., 0., 0., 1.1, 0.], [1.3, .9, .7],
                  [1., 1., 1.], [0, 1, 2])
nthread = 6
gate = threading.Barrier(nthread)
first, later = [None] * nthread, [None] * nthread

def work(t):
    with ecgpu.Context(0) as c:
        gate.wait()
        first[t] = c.int3c2e(ao, fit)
        later[t] = c.int3c2e(ao, fit)

threads = [threading.Thread(target=work, args=(t,)) for t in range(nthread)]
for t in threads: t.start()
for t in threads: t.join()
assert np.isfinite(later[0]).all() and np.abs(later[0]).max() > 0
for x in first + later:
    assert x is not None and np.array_equal(x, later[0])
"""


def test_first_integrals_of_a_process_in_several_contexts():
    src = PROGRAM.format(root=ROOT, pkg=os.path.join(ROOT, "elemco.jl_b200"))
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
