"""The rules for the ladder's a-blocks (csrc/ladder_blocks.h), compiled for the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "elemco.jl_b200", "csrc")


def _table(tmp_path, expr, nv):
    """expr(v) for v = 1 .. nv."""
    src = tmp_path / "t.cpp"
    src.write_text('#include <cstdio>\n#include "ladder_blocks.h"\nint main() {\n'
                   f"  for (long v = 1; v <= {nv}; ++v) printf(\"%ld\\n\", (long)({expr}));\n}}\n")
    exe = tmp_path / "t"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)])
    out = subprocess.check_output([str(exe)], text=True).split()
    return [None] + [int(x) for x in out]


def test_blocks_start_on_even_orbitals(tmp_path):
    """So that the rows of B a block reads start on 16 bytes; a block of one orbital,
    beyond 2 GiB of V an orbital pair row, is the exception."""
    na = _table(tmp_path, "ecg::ladder_na(5, v, 3 * v)", 700)
    for v in range(1, 701):
        assert 1 <= na[v] <= v
        assert na[v] == v or na[v] % 2 == 0 or na[v] == 1, (v, na[v])
        assert na[v] == 1 or na[v] * v ** 3 <= 1 << 28
        if v <= 508:  # two orbitals of V fit 2 GiB
            assert na[v] > 1 or v == 1


def test_blocks_fit_the_workspace(tmp_path):
    """What a block needs beside the callers' matrices is in the workspace, whose size
    goes by an eighth of the virtual space; blocks are as large as that allows."""
    for no, nq in ((1, 3), (2, 400), (7, 90), (40, 200), (3, 2000)):
        na = _table(tmp_path, f"ecg::ladder_na({no}, v, {nq})", 400)
        free = _table(tmp_path, f"ecg::system_workspace({no}, v, {nq}) - {no}L*{no}*{no}*{no} - "
                      f"4*(v + {no})*(v + {no}) - ecg::ladder_need({no}, v, {nq}, "
                      f"ecg::ladder_na({no}, v, {nq}))", 400)
        eighth = _table(tmp_path, "ecg::ladder_eighth(v)", 400)
        for v in range(1, 401):
            assert free[v] >= 0, (no, v, nq)
            assert na[v] == v or na[v] == 1 or na[v] % 2 == 0
            even = max(1, eighth[v] - eighth[v] % 2)
            assert -(-v // na[v]) <= -(-v // even), (no, v, nq)
