"""The three pattern kernels at the lengths and patterns where the rule turns from one to the other: the dense
kernel's columns that end inside a lane, a row or an item (it takes columns of 1.5, 3 or 40 MB and more), halves in
runs, which are gathered, and patterns that select everything, copied. Bit for bit against the CPU oracle, on
both sides of each line. Needs a B200."""
from __future__ import annotations

import pytest

from test_pattern_dense_gpu import _check

pytestmark = pytest.mark.gpu

MB = 1 << 20
DENSE = {1: 3 * MB, 2: 3 * MB // 2, 4: 3 * MB, 8: 40 * MB}  # payload bytes up to which a column is gathered
SCATTERED = [(0b10110010, 8), (0x7FFFFFFF, 32), (0b101, 3), (0b1010101, 13)]


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_dense_ends(cuda, oracle, w):
    ends = (0, 1, 32 // w - 1, 1024 // w + 1, 4096 // w - 1, 4096 // w, 3 * 4096 // w + 5, 131072 // w + 125)
    for i, extra in enumerate(ends if w < 8 else ends[1::3]):
        for pattern, length in (SCATTERED if w < 8 else SCATTERED[1:2] + [(0b1110111, 7)]):
            _check(oracle, w, DENSE[w] // w + extra, pattern, length, 0, i % 3)
            _check(oracle, w, DENSE[w] // w + extra, pattern, length, 16 // w, 0)  # a multiple of 16 bytes, not of 32


def test_half_of_8_byte_elements(cuda, oracle):
    for n in (96 * MB // 8, 96 * MB // 8 + 1):
        for pattern, length in SCATTERED[::2]:
            _check(oracle, 8, n, pattern, length, 0, 1)


@pytest.mark.parametrize("w", [2, 4, 8])
def test_halves_in_runs(cuda, oracle, w):
    for pattern, length in ((0x0000FFFF, 32), (0xFFFF0000, 32), (0xFF, 16), (0xF, 8), (0xFF00FF00, 32), (0x80007FFF, 32)):
        for n in (DENSE[min(w, 4)] // w + 77, 3_000_001):
            _check(oracle, w, n, pattern, length, 0, 1)


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_everything(cuda, oracle, w):
    for pattern, length in ((1, 1), (0x1FFFF, 17), (0xFFFFFFFF, 32)):
        for n in (1, 16 // w - 1 or 1, 16 // w + 1, 1000, 4096 // w * 4 + 1, 148 * 8 * 256 * 4 * 16 // w + 3, 1_000_003):
            _check(oracle, w, n, pattern, length, 0, 0)
        for n in (1000, 300_007):
            _check(oracle, w, n, pattern, length, 16 // w, 0)
            _check(oracle, w, n, pattern, length, 1, 0)  # inside a 16-byte group: gathered
            _check(oracle, w, n, pattern, length, 0, 1)


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_gathers_of_several_rounds(cuda, oracle, w):
    # unaligned, so gathered: a resident grid of 16 blocks per SM with 8 warps of 8 runs, once and once more
    outputs = 148 * 16 * 8 * 8 * max(128 // w, 32)
    for pattern, length in ((0b101, 3), (0b1110111, 7)):
        n = outputs // bin(pattern).count("1") * length
        for extra in (0, 1, n // 2 + 13):
            _check(oracle, w, n + extra, pattern, length, 1, 1)
