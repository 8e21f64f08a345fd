"""The 3-pass writeout by independent warps where it can go wrong: columns that end inside a
lane, a row, an item (4 KB of payload) or a unit, and columns, masks and outputs that start
inside a 16-byte group (AUTO takes them to this writeout). Bit for bit against the CPU oracle, and
nothing outside the output range is written. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, from_dev, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu

ITEM = 4096  # payload bytes
UNIT = 131072


def _column(n, w, seed, kind):
    rng = np.random.default_rng(seed)
    payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
    words = (n + 31) // 32
    if kind == "half":
        mask = rng.integers(0, 1 << 32, size=words, dtype=np.uint64).astype(np.uint32)
    elif kind == "full":  # bits past n are set too
        mask = np.full(words, 0xFFFFFFFF, np.uint32)
    else:  # runs of empty and full words, a few bits here and there
        mask = np.where(rng.integers(0, 3, words) == 0, 0xFFFFFFFF, 0).astype(np.uint32)
        mask ^= np.uint32(1) << rng.integers(0, 32, words).astype(np.uint32)
    return payload, mask


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("kind", ["half", "full", "mixed"])
def test_ragged_ends(cuda, oracle, w, kind):
    for nbytes in (w, 32, 32 + w, 1024 - w, 1024 + w, ITEM - w, ITEM, ITEM + w, 3 * ITEM + 40, UNIT - w, UNIT + 32 + w,
                   5 * UNIT + 3 * ITEM + 1000):
        n = max(1, nbytes // w)
        payload, mask = _column(n, w, n, kind)
        for chunk in (128, 4096 // w, 4096):
            check_against_oracle(oracle, payload, mask, n, "3pass", chunk_length=chunk)


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_unaligned_pointers(cuda, oracle, w):
    """Every phase of the payload within 16 bytes, of the mask within 4 words, of the output."""
    import torch
    import gpu_compressstore2_b200 as cs

    guard = 64
    for case, (n, kind) in enumerate(((1, "full"), (16 // w + 1, "full"), (1000, "half"), (ITEM // w + 5, "mixed"),
                                      (2 * UNIT // w + 999, "half"), (300_000, "sparse"))):
        payload, mask = _column(n, w, n + w, "mixed" if kind == "sparse" else kind)
        if kind == "sparse":
            mask = (mask & 1) * (np.arange(len(mask)) % 7 == 0).astype(np.uint32)
        exp = oracle.compact(payload, mask, n)
        for i in range(max(16 // w, 4)):
            in_off, mask_off, out_off = i, i % 4, (3 * i + case) % (16 // w + 1)
            d_in = to_dev(np.concatenate([np.zeros(in_off, UNSIGNED[w]), payload]))[in_off:]
            d_mask = to_dev(np.concatenate([np.full(mask_off, 0xFFFFFFFF, np.uint32), mask]))[mask_off:]
            d_out = dev_empty(out_off + n + guard, w, fill=0xAB)
            d_count = torch.full((1,), -7, dtype=torch.int64, device="cuda")
            cs.compressstore(d_in, d_mask, d_out[out_off:], n, d_count)
            torch.cuda.synchronize()
            k = int(d_count.item())
            out = from_dev(d_out, w)
            what = (w, n, in_off, mask_off, out_off)
            assert k == len(exp), what
            assert np.array_equal(out[out_off:out_off + k], exp), what
            rest = np.concatenate([out[:out_off], out[out_off + k:]]).view(np.uint8)
            assert np.all(rest == 0xAB), what


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_long_dense_column(cuda, oracle, w):
    """Many items per warp with 7 of 8 elements selected (the throttled grid of 4 and 8 bytes), a
    stretch of full words (the swizzled stage) and an empty one."""
    n = (8 * 148 * 3 * 8 * ITEM + 3 * UNIT) // w + 77
    rng = np.random.default_rng(w)
    words = (n + 31) // 32
    mask = np.zeros(words, np.uint32)
    for _ in range(3):
        mask |= rng.integers(0, 1 << 32, size=words, dtype=np.uint64).astype(np.uint32)
    mask[words // 3:words // 3 + words // 20] = 0xFFFFFFFF
    mask[words // 2:words // 2 + 3000] = 0
    payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
    check_against_oracle(oracle, payload, mask, n, "3pass", chunk_length=4096 // w)
