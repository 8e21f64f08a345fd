"""Chunks longer than the writeout's items (4 KB of payload): items at every place within a chunk, columns
that end in a chunk's first, middle and last item, masks and payloads inside a 16-byte group, sparse
units among dense ones. Bit for bit against the CPU oracle. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, from_dev, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu

ITEM = 4096


def _column(n, w, seed):
    """Stretches of 300 words: half, all, nothing, one in 64 selected; bits past n are set too."""
    rng = np.random.default_rng(seed)
    mask = rng.integers(0, 1 << 32, size=(n + 31) // 32, dtype=np.uint64).astype(np.uint32)
    kind = (np.arange(len(mask)) // 300) % 4
    mask[kind == 1] = 0xFFFFFFFF
    mask[kind == 2] = 0
    mask[kind == 3] = np.uint32(1) << (mask[kind == 3] & 31) * (mask[kind == 3] >> 31)
    return rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w]), mask


def _lengths(w, chunk):
    item = ITEM // w
    return [chunk - 1, chunk, chunk + 1, chunk + item + 1, 2 * chunk - item // 2, 40 * chunk + item - 3,
            3 * (131072 // w) + chunk // 2 + 5, 2_000_003]


@pytest.mark.parametrize("w,chunk", [(2, 4096), (4, 2048), (4, 4096), (8, 1024), (8, 2048), (8, 4096)])
def test_items_inside_chunks(cuda, oracle, w, chunk):
    import torch
    import gpu_compressstore2_b200 as cs

    for n in _lengths(w, chunk):
        payload, mask = _column(n, w, n)
        check_against_oracle(oracle, payload, mask, n, "3pass", chunk_length=chunk)
        exp = oracle.compact(payload, mask, n)
        b = cs.lib().cs_tune_size_bucket(n)
        assert cs.lib().cs_tune_set(w, b, cs.ALGO_3PASS, chunk) == 0  # AUTO takes unaligned pointers
        try:
            for in_off, mask_off in ((0, 1), (1, 0), (16 // w - 1, 3)):
                d_in = to_dev(np.concatenate([payload[:1].repeat(in_off), payload]))[in_off:]
                d_mask = to_dev(np.concatenate([np.full(mask_off, 0xFFFFFFFF, np.uint32), mask]))[mask_off:]
                d_out = dev_empty(n + 8, w, fill=0xAB)
                d_count = torch.zeros(1, dtype=torch.int64, device="cuda")
                cs.compressstore(d_in, d_mask, d_out, n, d_count)
                out = from_dev(d_out, w)
                assert int(d_count.item()) == len(exp), (n, in_off, mask_off)
                assert np.array_equal(out[:len(exp)], exp), (n, in_off, mask_off)
                assert np.all(out[len(exp):].view(np.uint8) == 0xAB), (n, in_off, mask_off)
        finally:
            cs.lib().cs_tune_set(w, b, cs.ALGO_AUTO, 1024)
    cs.lib().cs_tune_load(str(cs._lib.TUNE_TABLE).encode())
