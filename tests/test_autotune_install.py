"""A rebuilt tuning table keeps the library's choice by length in the two buckets in which the forms
change places: 4-byte columns of 2^24 .. 2^26 elements, 8-byte ones of 2^22 .. 2^24."""
from __future__ import annotations

import ctypes


def _form(L, w, n):
    algo, chunk = ctypes.c_int32(), ctypes.c_uint32()
    assert L.cs_tune_get(w, n, ctypes.byref(algo), ctypes.byref(chunk)) == 0
    return algo.value


def test_rebuilt_table_keeps_the_lengths(tmp_path):
    import gpu_compressstore2_b200 as cs
    from gpu_compressstore2_b200 import autotune

    L = cs.lib()
    line = 76 << 20  # bytes
    try:
        # as tune() returns them: every bucket measured, one form for each
        sel = {s: (cs.ALGO_3PASS, 1024) for s in range(5)}
        autotune.install({(w, b): (cs.ALGO_3PASS, 1024, {}, sel) for w in (1, 2, 4, 8) for b in (11, 12)})
        out = tmp_path / "t.txt"
        autotune.save(out)
        for when in ("as installed", "as loaded"):
            if when == "as loaded":
                for w in (1, 2, 4, 8):
                    for b in (11, 12):
                        L.cs_tune_set(w, b, cs.ALGO_AUTO, 0)
                assert autotune.load(out)
            for w in (4, 8):
                assert _form(L, w, line // w) == cs.ALGO_1PASS, (when, w)
                assert _form(L, w, line // w + 1) == cs.ALGO_3PASS, (when, w)
            for w, n in ((4, 1 << 22), (8, 1 << 24), (1, 1 << 24), (2, 1 << 22)):
                assert _form(L, w, n) == cs.ALGO_3PASS, (when, w, n)
        words = [ln.split()[:2] for ln in out.read_text().splitlines() if ln[:1].isdigit()]
        assert ["4", "12"] not in words and ["8", "11"] not in words and ["4", "11"] in words
    finally:
        for w in (1, 2, 4, 8):
            for b in (11, 12):
                L.cs_tune_set(w, b, cs.ALGO_AUTO, 0)
                for s in range(5):
                    L.cs_tune_sel_set(w, b, s, cs.ALGO_AUTO, 0)
        assert L.cs_tune_load(str(cs._lib.TUNE_TABLE).encode()) == 0
