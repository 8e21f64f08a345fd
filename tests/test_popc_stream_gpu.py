"""The counting pass over long masks and plans of many blocks, where it can go wrong: last blocks of
every kind (words past the last 16-byte group, bits past the last word, masks that start inside a
group), plans with more blocks than the passes keep in shared memory at once. Bit for bit against
the CPU oracle. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import from_dev, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu

BLOCK = 1 << 18


def _run_plan(oracle, sizes, w):
    """Columns of the given sizes in one 3-pass plan."""
    import torch
    import gpu_compressstore2_b200 as cs

    rng = np.random.default_rng(len(sizes) + w)
    words = [(n + 31) // 32 for n in sizes]
    at_m = np.concatenate([[0], np.cumsum([(k + 3) // 4 * 4 for k in words])])
    at_p = np.concatenate([[0], np.cumsum([(n + 15) // 16 * 16 for n in sizes])])
    mask = rng.integers(0, 1 << 32, size=int(at_m[-1]) + 8, dtype=np.uint64).astype(np.uint32)
    payload = oracle.payload(int(at_p[-1]), w, 7)
    d_mask, d_in = to_dev(mask), to_dev(payload)
    d_out = torch.zeros_like(d_in)
    counts = torch.full((len(sizes),), -5, dtype=torch.int64, device="cuda")
    cols = [(d_in[at_p[i]:at_p[i] + n], d_mask[at_m[i]:at_m[i] + words[i]], d_out[at_p[i]:at_p[i] + n], n, counts[i:i + 1])
            for i, n in enumerate(sizes)]
    plan = cs.Batch(cols, algo=cs.ALGO_3PASS)
    for _ in range(2):
        plan.run()
    torch.cuda.synchronize()
    got, out = counts.cpu().numpy(), from_dev(d_out, w)
    for i, n in enumerate(sizes):
        a = at_p[i]
        exp = oracle.compact(payload[a:a + n], mask[at_m[i]:at_m[i] + words[i]], n)
        assert got[i] == len(exp), (i, n)
        assert np.array_equal(out[a:a + len(exp)], exp), (i, n)
        assert not out[a + len(exp):a + n].any(), (i, n)


EDGES = [1, 31, 32, 33, 95, 96, 97, 127, 128, 129, 161, 4095, 4096, 4097, 32768 + 130, BLOCK - 129, BLOCK - 1, BLOCK, BLOCK + 1,
         BLOCK + 160, 2 * BLOCK + 32768 - 33]


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("repeat", [1, 34])
def test_last_blocks(cuda, oracle, w, repeat):
    _run_plan(oracle, EDGES * repeat, w)


@pytest.mark.parametrize("columns", [8180, 8193, 30001])
def test_many_blocks(cuda, oracle, columns):
    """Past 8192 blocks the column prefixes are made in memory; past 32 blocks per CTA the table of
    blocks is refilled."""
    _run_plan(oracle, [1 + (i * 37) % 200 for i in range(columns - 2)] + [BLOCK + 77, 3], 1)


@pytest.mark.parametrize("chunk", [128, 512, 4096])
def test_long_column(cuda, oracle, chunk):
    for n, shift in ((600 * BLOCK + 1000, 0), (600 * BLOCK + 1000, 1)):
        import torch
        import gpu_compressstore2_b200 as cs

        rng = np.random.default_rng(n + chunk)
        mask = rng.integers(0, 1 << 32, size=(n + 31) // 32 + 4, dtype=np.uint64).astype(np.uint32)[shift:]
        payload = rng.integers(0, 256, size=n, dtype=np.uint8)
        if shift == 0:
            check_against_oracle(oracle, payload, mask[:(n + 31) // 32], n, "3pass", chunk_length=chunk)
            continue
        d_mask = to_dev(np.concatenate([np.zeros(shift, np.uint32), mask]))[shift:]
        d_in = to_dev(payload)
        d_out = torch.zeros_like(d_in)
        count = torch.zeros(1, dtype=torch.int64, device="cuda")
        cs.compressstore(d_in, d_mask, d_out, n, count)
        exp = oracle.compact(payload, mask[:(n + 31) // 32], n)
        assert count.item() == len(exp)
        assert np.array_equal(from_dev(d_out, 1)[:len(exp)], exp)
