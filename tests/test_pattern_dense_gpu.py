"""Both pattern kernels where their work split can go wrong: columns that end inside a lane, a row,
an item or a run, several items per warp, inputs and outputs inside a 16-byte group, odd and even
numbers selected per period, shares on both sides of the rule that picks the kernel. Bit for bit
against the CPU oracle. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, from_dev, to_dev

pytestmark = pytest.mark.gpu

PATTERNS = [(0b1, 1), (0b10, 2), (0b101, 5), (0b11, 3), (0b110, 6), (0b1, 8), (0b10110010, 8), (0b1011011, 10),
            (0x7FFFFFFF, 32), (0x80000001, 32), (0b1010101, 31)]


def _check(oracle, w, n, pattern, length, in_off, out_off):
    import torch
    import gpu_compressstore2_b200 as cs

    rng = np.random.default_rng(n + length)
    payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
    exp = oracle.compact(payload, oracle.mask_pattern(n, pattern, length), n)
    d_in = to_dev(np.concatenate([np.zeros(in_off, UNSIGNED[w]), payload]))[in_off:]
    d_out = dev_empty(out_off + n + 64, w, fill=0xAB)
    d_count = torch.full((1,), -7, dtype=torch.int64, device="cuda")
    cs.compressstore_pattern(d_in, d_out[out_off:], n, pattern, length, d_count)
    torch.cuda.synchronize()
    k, out = int(d_count.item()), from_dev(d_out, w)
    what = (w, n, bin(pattern), length, in_off, out_off)
    assert k == len(exp), what
    assert np.array_equal(out[out_off:out_off + k], exp), what
    assert np.all(np.concatenate([out[:out_off], out[out_off + k:]]).view(np.uint8) == 0xAB), what


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_pattern_ends_and_phases(cuda, oracle, w):
    for pattern, length in PATTERNS:
        for nbytes in (w, 32 - w if w < 32 else 32, 32 + w, 1024 - w, 4096 - w, 4096, 4096 + w, 3 * 4096 + 40, 131072 + 1000):
            n = max(1, nbytes // w)
            _check(oracle, w, n, pattern, length, 0, 0)
            _check(oracle, w, n, pattern, length, 16 // w, 3)     # a multiple of 16 bytes, not of 32
            _check(oracle, w, n, pattern, length, 1, 16 // w + 1)  # inside a 16-byte group


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_pattern_many_items_per_warp(cuda, oracle, w):
    n = 148 * 3 * 8 * 4096 * 2 // w + 12345
    for pattern, length in ((0b101, 5), (0b10110010, 8), (0x7FFFFFFF, 32), (0b1, 16)):
        _check(oracle, w, n, pattern, length, 0, 1)
