"""The 1-pass form in slices of 32 KB where its split can go wrong: one slice, a slice for every CTA
and one more, several per CTA, columns that end inside a lane or an item, masks and outputs inside a
16-byte group, items with nothing, a few, nearly all selected. Bit for bit against the CPU oracle.
Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, dev_empty, from_dev, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu

SLICE = 32768
CTAS = 148 * 3


def _mask(n, w, rng):
    """Item by item (4 KB of payload): nothing, a few, 1/16 and one more, half, nearly all, all."""
    bits = np.zeros(n, dtype=np.uint8)
    per = 4096 // w
    for i, e0 in enumerate(range(0, n, per)):
        size = min(per, n - e0)
        k = (0, 3, 64, 65, size // 2, size - 1, size)[i % 7]
        bits[e0 + rng.permutation(size)[:min(k, size)]] = 1
    return np.packbits(np.concatenate([bits, np.zeros(-n % 32, np.uint8)]), bitorder="little").view(np.uint32)


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("slices", [1, 2, CTAS, CTAS + 1, 8 * 148])
def test_onepass_slices(cuda, oracle, w, slices):
    rng = np.random.default_rng(slices + w)
    for extra in (0, -1) if slices > 2 else (0, -1, -4096 // w + 3, 1 - SLICE // w):
        n = slices * SLICE // w + extra
        payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
        check_against_oracle(oracle, payload, _mask(n, w, rng), n, "1pass")


@pytest.mark.parametrize("w", [1, 2, 4, 8])
def test_auto_unaligned_mask_and_output(cuda, oracle, w):
    """Short columns whose payload is 16-byte aligned and whose mask and output are not."""
    import torch
    import gpu_compressstore2_b200 as cs

    rng = np.random.default_rng(w)
    n = 3 * SLICE // w + 77
    payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
    mask = _mask(n, w, rng)
    exp = oracle.compact(payload, mask, n)
    for mask_off, out_off in ((1, 0), (0, 1), (3, 16 // w + 1)):
        d_mask = to_dev(np.concatenate([np.full(mask_off, 0xFFFFFFFF, np.uint32), mask]))[mask_off:]
        d_out = dev_empty(out_off + n + 64, w, fill=0xAB)
        d_count = torch.zeros(1, dtype=torch.int64, device="cuda")
        before = cs.launch_count()
        cs.compressstore(to_dev(payload), d_mask, d_out[out_off:], n, d_count)
        torch.cuda.synchronize()
        assert cs.launch_count() - before <= 3
        k, out = int(d_count.item()), from_dev(d_out, w)
        assert k == len(exp)
        assert np.array_equal(out[out_off:out_off + k], exp)
        assert np.all(np.concatenate([out[:out_off], out[out_off + k:]]).view(np.uint8) == 0xAB)


@pytest.mark.parametrize("w,n", [(4, 18 * 148 * 8192), (4, 18 * 148 * 8192 + 1), (4, (76 << 20) // 4), (4, (76 << 20) // 4 + 1),
                                 (8, (76 << 20) // 8), (8, (76 << 20) // 8 + 1), (4, (1 << 24) + 4099)])
def test_where_the_forms_change(cuda, oracle, w, n):
    """Both sides of the lines between slices, the other 1-pass kernel and the 3-pass form."""
    import gpu_compressstore2_b200 as cs

    rng = np.random.default_rng(n)
    payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w])
    mask = rng.integers(0, 1 << 32, size=(n + 31) // 32, dtype=np.uint64).astype(np.uint32)
    check_against_oracle(oracle, payload, mask, n, "1pass")
    check_against_oracle(oracle, payload, mask, n, "auto")  # its scratch sized
    before = cs.launch_count()
    check_against_oracle(oracle, payload, mask, n, "auto")
    assert (cs.launch_count() - before == 1) == (n * w <= 76 << 20)
