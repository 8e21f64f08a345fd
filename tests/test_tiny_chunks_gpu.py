"""Chunks of 32 and 64 elements, whose columns have no pass that counts sparse groups: results against the
CPU oracle on both sides of the length from which units are gathered, and short dense columns are not
gathered one element after another. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("chunk", [32, 64])
def test_results(cuda, oracle, w, chunk):
    rng = np.random.default_rng(w)
    for n in (1, 4101, 131072 // w + 7, 255 * 16384, 256 * 16384 + 5):
        payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
        for p in (0.01, 0.95):
            check_against_oracle(oracle, payload, oracle.mask_bernoulli(n, p, n), n, "3pass", chunk_length=chunk)


def test_short_dense_column(cuda, oracle):
    import torch
    import gpu_compressstore2_b200 as cs

    n = 4101
    x, mask, out = dev_empty(n, 1, fill=1), to_dev(oracle.mask_bernoulli(n, 0.95, 1)), dev_empty(n, 1)
    count = torch.zeros(1, dtype=torch.int64, device="cuda")

    def us(chunk):
        best = float("inf")
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                cs.compressstore(x, mask, out, n, count, algo=cs.ALGO_3PASS, chunk_length=chunk)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 50)
        return best

    short, ordinary = us(32), us(128)  # three launches, two
    print(f"{short:.1f} {ordinary:.1f} us")
    assert short < 3.5 * ordinary
