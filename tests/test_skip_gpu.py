"""cs_config.skip = 2 loads whole tiles whether or not anything in them is selected: with an empty mask
a call reads its whole payload, and so takes several times as long as one that skips. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, from_dev, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu


def _us(call, reps=10):
    """Fastest of `reps` calls, on the device."""
    import torch

    best = float("inf")
    for _ in range(3 + reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        call()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


# 512 MB of payload, which take 80 us to read at the copy rate, and 16 to 64 MB of mask
@pytest.mark.parametrize("w,algo,chunk", [(1, "1PASS", 1024), (2, "1PASS", 1024), (4, "3PASS", 1024), (8, "3PASS", 4096)])
def test_skip_2_reads_the_payload(cuda, w, algo, chunk):
    import torch
    import gpu_compressstore2_b200 as cs

    n = (512 << 20) // w
    d_in, d_out = dev_empty(n, w, fill=1), dev_empty(n, w, fill=0)
    d_mask = torch.zeros(n // 32, dtype=torch.int32, device="cuda")
    d_count = torch.zeros(1, dtype=torch.int64, device="cuda")

    def call(skip):
        cs.compressstore(d_in, d_mask, d_out, n, d_count, algo=getattr(cs, "ALGO_" + algo), chunk_length=chunk, skip=skip)

    skipping, whole = _us(lambda: call(1)), _us(lambda: call(2))
    print(f"{w} {algo}: {skipping:.1f} {whole:.1f} us")
    assert whole > 75.0 and whole > 1.4 * skipping
    assert int(d_count.item()) == 0


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_skip_2_results(cuda, oracle, w):
    """Every form, short and long columns, aligned or not, with skip = 2."""
    import torch
    import gpu_compressstore2_b200 as cs

    rng = np.random.default_rng(w)
    for n in (1000, 300_000, 5_000_011):
        payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
        for p in (0.01, 0.5):
            mask = oracle.mask_bernoulli(n, p, n)
            for algo, chunk in (("1pass", 1024), ("3pass", 512), ("3pass", 4096), ("auto", 0)):
                check_against_oracle(oracle, payload, mask, n, algo, chunk_length=chunk, skip=2)
            exp = oracle.compact(payload, mask, n)
            src = to_dev(np.concatenate([payload[:1], payload]))[1:]
            out, count = dev_empty(n, w), torch.zeros(1, dtype=torch.int64, device="cuda")
            cs.compressstore(src, to_dev(mask), out, n, count, skip=2)
            assert int(count.item()) == len(exp)
            assert np.array_equal(from_dev(out, w)[:len(exp)], exp)
