"""What a CTA of the 1-pass form in slices takes for another slice's total. The ticket of slice 0 is
given away by hand, so nobody publishes its total, and the workspace holds something else in its
place: the call reports an error and writes nothing, and the workspace works again afterwards. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev_empty, from_dev, to_dev
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu

AGG, POISON = 1, 3


def _refused(oracle, flag, value, status):
    import torch
    import gpu_compressstore2_b200 as cs

    n = 64 * 8192
    payload, mask = oracle.payload(n, 4, 1), oracle.mask_bernoulli(n, 0.5, 2)
    ws = cs.Workspace.for_call(n, 4, cs.make_config(cs.ALGO_1PASS))
    torch.cuda.synchronize()
    off = ws.ptr - ws.buf.data_ptr()
    words = ws.buf[off:off + ws.nbytes].view(torch.int64)
    words[2] = 1  # tile_counter = 1, done_counter = 0
    epoch = int(words[0]) >> 32
    words[32:] = epoch << 42 | flag << 40 | value
    d_out = dev_empty(n, 4, fill=0xCD)
    d_count = torch.zeros(1, dtype=torch.int64, device="cuda")
    cs.compressstore(to_dev(payload), to_dev(mask), d_out, n, d_count, algo=cs.ALGO_1PASS, timeout_ns=20_000_000,
                     workspace=ws)
    with pytest.raises(cs.CsError) as ei:
        ws.check()
    assert ei.value.status == status
    assert int(d_count.item()) == -1
    assert np.all(from_dev(d_out, 4).view(np.uint8) == 0xCD)
    check_against_oracle(oracle, payload, mask, n, "1pass", workspace=ws)


def test_another_flag_is_no_total(cuda, oracle):
    import gpu_compressstore2_b200 as cs

    _refused(oracle, POISON, 0, cs._lib.ERR_TIMEOUT)


def test_a_total_larger_than_a_slice(cuda, oracle):
    """It would lead past the end of the output."""
    import gpu_compressstore2_b200 as cs

    for value in (8193, 1 << 30, (1 << 32) - 1):
        _refused(oracle, AGG, value, cs._lib.ERR_INVALID_VALUE)
