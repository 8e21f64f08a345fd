"""The 1-pass form in slices does not depend on the chunk length: its totals fit every workspace, and
the form that a call takes is the same at every chunk length."""
from __future__ import annotations

import ctypes
import random

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, from_dev, to_dev

HEADER, SLICE = 256, 32768


@pytest.mark.parametrize("w,most", [(1, 1 << 40), (2, 1 << 40), (4, 18 * 148 * 8192), (8, 8 * 148 * 4096)])
def test_totals_fit_the_workspace(w, most):
    """Lengths up to those that run in slices (1- and 2-byte columns: all)."""
    import gpu_compressstore2_b200 as cs

    rng = random.Random(w)
    for n in [1, most - 1] + [int(2 ** rng.uniform(0, np.log2(most))) for _ in range(2000)]:
        for log2 in (5, 10, 16):
            cfg = cs.make_config(cs.ALGO_1PASS, 1 << log2)
            size = cs.lib().compressstore_workspace_size(n, w, ctypes.byref(cfg))
            assert HEADER + 8 * -(-n * w // SLICE) <= size, (n, log2)


@pytest.mark.gpu
@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("chunk", [0, 32, 65536])
def test_one_launch_at_every_chunk_length(cuda, oracle, w, chunk):
    """A mask and an output inside a 16-byte group, which slices take and the TMA kernel does not."""
    import torch
    import gpu_compressstore2_b200 as cs

    n = 300_000
    rng = np.random.default_rng(w)
    payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
    mask = oracle.mask_bernoulli(n, 0.5, w)
    exp = oracle.compact(payload, mask, n)
    L = cs.lib()
    b = L.cs_tune_size_bucket(n)
    assert L.cs_tune_set(w, b, cs.ALGO_1PASS, 1024) == 0
    try:
        d_in, d_mask = to_dev(payload), to_dev(np.concatenate([mask[:1], mask]))[1:]
        d_count = torch.zeros(1, dtype=torch.int64, device="cuda")
        for warm in (True, False):  # the scratch is sized by the first call
            d_out = dev_empty(n + 1, w, fill=0xAB)
            before = cs.launch_count()
            cs.compressstore(d_in, d_mask, d_out[1:], n, d_count, chunk_length=chunk)
            launches = cs.launch_count() - before
            assert warm or launches == 1, launches
            assert int(d_count.item()) == len(exp)
            got = from_dev(d_out, w)[1:]
            assert np.array_equal(got[:len(exp)], exp) and np.all(got[len(exp):].view(np.uint8) == 0xAB)
    finally:
        L.cs_tune_set(w, b, cs.ALGO_AUTO, 1024)
        L.cs_tune_load(str(cs._lib.TUNE_TABLE).encode())
