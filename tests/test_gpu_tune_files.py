"""Tuning files of earlier versions: FP64 entries that name TMA tiles of then (numbers 1
to 3) are left out, the others are used, and a saved table says whose numbers it has."""
import pytest

import ecgpu

pytestmark = pytest.mark.gpu


def _load(c, tmp_path, *lines):
    p = tmp_path / "t.txt"
    p.write_text("".join(x + "\n" for x in lines))
    return c.tune_load(p)


def test_entries_of_other_tiles_are_left_out(tmp_path):
    with ecgpu.Context(0) as c:
        _load(c, tmp_path, "dgemmt 1001 1 1 1 00 8")  # a first FP64 entry
        n = _load(c, tmp_path, "tc 1001 1 1 2 0 4")
        # 8 S + 4 + tile, TMA; 8 S + tile, cp.async
        assert _load(c, tmp_path, "dgemmt 1003 7 9 1 00 13", "dgemmt 1005 7 9 1 00 14",
                     "dgemmt 1007 7 9 1 00 31") == n
        assert _load(c, tmp_path, "dgemmt 1009 7 9 1 00 12", "dgemmt 1011 7 9 1 00 10") == n + 2
        assert _load(c, tmp_path, "dgemmt-tiles 2", "dgemmt 1003 7 9 1 00 13") == n + 3
        assert _load(c, tmp_path, "dgemmt-tiles 3", "dgemmt 1005 7 9 1 00 14") == n + 3
        p = tmp_path / "s.txt"
        assert c.tune_save(p) == n + 3
        text = p.read_text().splitlines()
        assert "dgemmt-tiles 2" in text and "dgemmt 1003 7 9 1 00 13" in text
        assert c.tune_load(p) == n + 3
