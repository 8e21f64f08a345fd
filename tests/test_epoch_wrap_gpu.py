"""The end of an epoch cycle (2^22 calls on one workspace), reached by setting the header's epoch:
afterwards nothing in the workspace reads as a status, neither marks of the call that ended the
cycle nor statuses that earlier calls left, and every form still equals the CPU oracle. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import UNSIGNED, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu

EPOCH_MIN, LAST = 128, (1 << 22) - 2
N_MAX = 5_000_000


def _header(ws):
    import torch

    off = ws.ptr - ws.buf.data_ptr()
    return ws.buf[off:off + ws.nbytes].view(torch.int32)


def _epoch(ws):
    import torch

    torch.cuda.synchronize()
    return int(_header(ws)[1])


def _status_words(ws):
    """Words after the header whose epoch field is a valid one."""
    words = _header(ws).cpu().numpy().view(np.uint64)[32:]
    return np.flatnonzero((words >> np.uint64(42)) >= EPOCH_MIN)


def _column(oracle, n, w, p, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, 256, size=n * w, dtype=np.uint8).view(UNSIGNED[w]), oracle.mask_bernoulli(n, p, seed)


# (form, chunk length) of the call that ends the cycle
@pytest.mark.parametrize("algo,chunk", [("3pass", 512), ("3pass", 4096), ("3pass", 64), ("naive", 32), ("1pass", 1024)])
@pytest.mark.parametrize("n", [1000, 300_000, N_MAX])
def test_no_status_outlives_the_cycle(cuda, oracle, algo, chunk, n):
    import gpu_compressstore2_b200 as cs

    ws = cs.Workspace.for_call(N_MAX, 8, cs.make_config(cs.ALGO_3PASS, 32))
    # statuses of both 1-pass kernels and of the scan, of several layouts
    for m, w, a, c in ((N_MAX, 8, "1pass", 1024), (4_000_000, 8, "1pass", 1024), (3_000_000, 4, "1pass", 1024),
                       (50_000, 1, "1pass", 4096), (N_MAX, 4, "naive", 32)):
        check_against_oracle(oracle, *_column(oracle, m, w, 0.5, m), m, a, chunk_length=c, workspace=ws)
    for p in (0.01, 0.5):
        _header(ws)[1] = LAST
        payload, mask = _column(oracle, n, 4, p, n)
        check_against_oracle(oracle, payload, mask, n, algo, chunk_length=chunk, workspace=ws)
        assert _epoch(ws) == EPOCH_MIN
        assert len(_status_words(ws)) == 0
        # the new cycle
        for a, c in (("1pass", 1024), ("3pass", chunk if chunk >= 128 else 1024), ("naive", 32), ("1pass", 1024)):
            check_against_oracle(oracle, payload, mask, n, a, chunk_length=c, workspace=ws)
        ws.check()
