"""Predicate compaction over columns of several slices per CTA: items with nothing, with a few
(gathered), with just more than that and with nearly all elements selected, a column that ends
inside a lane, and the mask output. Against numpy's own indexing. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev_empty, from_dev, to_dev, UNSIGNED

pytestmark = pytest.mark.gpu

TYPES = {0: np.uint8, 5: np.int16, 6: np.int32, 7: np.int64, 8: np.float32, 9: np.float64}
ITEM = 4096
FEW = 64


def _column(dt, n, rng):
    """1 where the element is to be selected by x >= 1, else 0; the share changes item by item."""
    per = ITEM // dt().itemsize
    x = np.zeros(n, dtype=dt)
    for i, e0 in enumerate(range(0, n, per)):
        size = min(per, n - e0)
        kind = i % 7
        if kind == 6:
            continue
        want = (1, FEW, FEW + 1, size // 2, size - 1, size)[kind]
        x[e0 + rng.permutation(size)[:min(want, size)]] = 1
    return x


@pytest.mark.parametrize("code", list(TYPES))
@pytest.mark.parametrize("slices", [1, 3, 148 * 3 * 5])
def test_slices(cuda, oracle, code, slices):
    import torch
    import gpu_compressstore2_b200 as cs

    dt = TYPES[code]
    w = dt().itemsize
    rng = np.random.default_rng(code + slices)
    for extra in (-1, 0, 13):
        if slices > 3 and extra != 13:
            continue
        n = slices * 8 * ITEM // w + extra
        x = _column(dt, n, rng)
        for op, a, b, sel in ((">=", 1, None, x >= 1), ("==", 0, None, x == 0), ("between", 1, 1, x == 1)):
            if slices > 3 and op != ">=":
                continue
            d_out = dev_empty(n + 32, w, fill=0xA5)
            d_mask = torch.full(((n + 31) // 32 + 4,), -1, dtype=torch.int32, device="cuda")
            d_count = torch.zeros(1, dtype=torch.int64, device="cuda")
            cs.compressstore_if(to_dev(x.view(UNSIGNED[w])), d_out, n, cs.predicate(op, a, b, elem_type=code), d_count,
                                d_mask_out=d_mask)
            torch.cuda.synchronize()
            k, got = int(d_count.item()), from_dev(d_out, w)
            assert k == int(sel.sum()), (dt, n, op)
            assert np.array_equal(got[:k], x[sel].view(UNSIGNED[w])), (dt, n, op)
            assert np.all(got[k:].view(np.uint8) == 0xA5), (dt, n, op)
            words = from_dev(d_mask, 4)
            bits = np.unpackbits(words[:(n + 31) // 32].view(np.uint8), bitorder="little")
            assert np.array_equal(bits[:n].astype(bool), sel) and not bits[n:].any(), (dt, n, op)
            assert np.all(words[(n + 31) // 32:] == 0xFFFFFFFF), (dt, n, op)
    cs.compressstore_check()
