"""The sparse gather of the 3-pass form where its work split can go wrong: units at exactly the
1/32 limit and one past it, clusters that fill a warp's index list several times over, whole
and quarter work items (columns of 2^22 elements and more), columns that end inside an item, chunks shorter than a group. Bit for
bit against the CPU oracle. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu

UNIT_BYTES = 131072
WHOLE_ITEMS_N = 148 * 64 // 4 * 16384 + 3 * 131072  # elements past which a warp takes whole items


def _mask(n, w, rng):
    """Per unit, in turn: empty; 1/32 of it selected in one run; the same scattered; one more
    than 1/32; a single last element; a thin random selection."""
    bits = np.zeros(n, dtype=np.uint8)
    unit = UNIT_BYTES // w
    most = unit // 32
    for i, u0 in enumerate(range(0, n, unit)):
        size = min(unit, n - u0)
        kind = i % 6
        if kind == 1:
            at = int(rng.integers(0, max(1, size - most)))
            bits[u0 + at:u0 + min(size, at + most)] = 1
        elif kind in (2, 3):
            k = min(size, most + (kind == 3))
            bits[u0 + rng.choice(size, k, replace=False)] = 1
        elif kind == 4:
            bits[u0 + size - 1] = 1
        elif kind == 5:
            bits[u0 + rng.integers(0, size, size // 1000 + 1)] = 1
    return np.packbits(np.concatenate([bits, np.zeros(-n % 32, np.uint8)]), bitorder="little").view(np.uint32)


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("n,chunk_length", [(16384 * 3 + 1, 1024), (16384 * 3 + 1, 4096), (131072 * 13 - 33, 1024),
                                            (131072 * 13 - 33, 4096), (131072 * 70 - 33, 1024), (WHOLE_ITEMS_N + 4097, 4096)])
def test_sparse_units(cuda, oracle, n, w, chunk_length):
    rng = np.random.default_rng(n + w)
    payload = rng.integers(0, 256, size=n * w, dtype=np.uint8).view({1: np.uint8, 2: np.uint16, 4: np.uint32,
                                                                     8: np.uint64}[w])
    check_against_oracle(oracle, payload, _mask(n, w, rng), n, "3pass", chunk_length=chunk_length)
