"""The bounded look-back of the TMA 1-pass kernel, which serves long 4- and 8-byte columns, skip = 2 and
the 1-pass columns of plans: a unit that nobody processes leaves its successors waiting. They give up,
the call reports the error and writes nothing, and the workspace works again. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev_empty, from_dev, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu


# one-tile units, units of four tiles, and the deeper ring of 16 units per SM and more
@pytest.mark.parametrize("n,skip", [(64 * 8192, 2), (152 * 32768, 2), (16 * 152 * 32768, 0)])
def test_lookback_timeout(cuda, oracle, n, skip):
    import torch
    import gpu_compressstore2_b200 as cs

    payload, mask = oracle.payload(n, 4, 1), oracle.mask_bernoulli(n, 0.5, 2)
    ws = cs.Workspace.for_call(n, 4, cs.make_config(cs.ALGO_1PASS))
    torch.cuda.synchronize()
    off = ws.ptr - ws.buf.data_ptr()
    ws.buf[off + 16:off + 20].view(torch.int32).fill_(1)  # tile_counter = 1: unit 0 is never taken
    d_out = dev_empty(n, 4, fill=0xCD)
    d_count = torch.zeros(1, dtype=torch.int64, device="cuda")
    cs.compressstore(to_dev(payload), to_dev(mask), d_out, n, d_count, algo=cs.ALGO_1PASS, skip=skip,
                     timeout_ns=20_000_000, workspace=ws)
    with pytest.raises(cs.CsError) as ei:
        ws.check()
    assert ei.value.status == cs._lib.ERR_TIMEOUT
    assert int(d_count.item()) == -1
    assert np.all(from_dev(d_out, 4).view(np.uint8) == 0xCD)
    check_against_oracle(oracle, payload, mask, n, "1pass", workspace=ws, skip=skip)
    ws.check()
