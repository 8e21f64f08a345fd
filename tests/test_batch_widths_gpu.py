"""A long sparse column beside short columns of every width in one plan: bit for bit against the CPU
oracle, and the short columns' launches do not walk the long one's items. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, from_dev, to_dev

pytestmark = pytest.mark.gpu

SMALL = [(300_000, 4, 0.5), (1_000_000, 1, 0.004), (70_001, 8, 0.01), (5000, 2, 0.5), (300_000, 4, 0.01), (70_001, 8, 0.5)]


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("at", [0, 3, 6])
def test_results(cuda, oracle, w, at):
    """The long column first, in the middle and last in the plan."""
    import torch
    import gpu_compressstore2_b200 as cs

    n = 12_345_678
    rng = np.random.default_rng(w + at)
    specs = SMALL[:at] + [(n, w, 0.01)] + SMALL[at:]
    host = [(rng.integers(0, 256, size=m * v, dtype=np.uint8).view(UNSIGNED[v]), oracle.mask_bernoulli(m, p, i)) for i, (m, v, p) in enumerate(specs)]
    counts = torch.zeros(len(specs), dtype=torch.int64, device="cuda")
    outs = [dev_empty(m + 8, v, fill=0xAB) for m, v, _ in specs]
    plan = cs.Batch([(to_dev(x), to_dev(np.concatenate([k, np.zeros(-len(k) % 4, np.uint32)])), o, m, counts[i:i + 1])
                     for i, ((x, k), o, (m, _, _)) in enumerate(zip(host, outs, specs))], algo=cs.ALGO_3PASS)
    plan.run()
    plan.check()
    for (x, k), o, (m, v, _), c in zip(host, outs, specs, counts.tolist()):
        exp, got = oracle.compact(x, k, m), from_dev(o, v)
        assert c == len(exp)
        assert np.array_equal(got[:c], exp) and np.all(got[c:].view(np.uint8) == 0xAB)
    plan.close()


def test_short_columns_cost_little(cuda):
    import torch
    import gpu_compressstore2_b200 as cs

    def plan_us(specs):
        keep, cols = [], []
        for i, (n, w, p) in enumerate(specs):
            x, mask = dev_empty(n, w, fill=i), torch.empty((n + 127) // 128 * 4, dtype=torch.int32, device="cuda")
            cs.gen_mask_bernoulli(mask, n, p, i)
            cols.append((x, mask, dev_empty(n, w), n, torch.zeros(1, dtype=torch.int64, device="cuda")))
        plan = cs.Batch(cols, algo=cs.ALGO_3PASS)
        best = float("inf")
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                plan.run()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 100)
        plan.check()
        plan.close()
        return best

    long = (1 << 28, 1, 0.01)
    alone, beside = plan_us([long]), plan_us([long] + SMALL)
    print(f"{alone:.1f} {beside:.1f} us")
    assert beside < 2 * alone  # three more launches of 5 to 8 us each
