"""When a long column's writeout gathers its sparse units: from one sparse 16K-element group in 12 on,
wherever they lie. Whether it did is read from the workspace's header. Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, GROUP_WORDS = 1 << 28, 512  # two or three blocks of pass 1 + 2 for each of its CTAs


@pytest.mark.parametrize("every,gathers", [(1, True), (8, True), (10, True), (11, True), (13, False), (16, False), (0, False)])
@pytest.mark.parametrize("w", [4, 8])
def test_evenly_spread_sparse_groups(cuda, every, gathers, w):
    import torch
    import gpu_compressstore2_b200 as cs

    groups = torch.full((N // 32 // GROUP_WORDS, GROUP_WORDS), 0x55555555, dtype=torch.int32, device="cuda")
    if every:
        groups[::every] = 0
    d_mask = groups.view(-1)
    dt = {4: torch.int32, 8: torch.int64}[w]
    d_in = torch.arange(N, dtype=dt, device="cuda")
    d_out = torch.empty_like(d_in)
    d_count = torch.zeros(1, dtype=torch.int64, device="cuda")
    ws = cs.Workspace.for_call(N, w, cs.make_config(cs.ALGO_3PASS, 512))
    cs.compressstore(d_in, d_mask, d_out, N, d_count, algo=cs.ALGO_3PASS, chunk_length=512, workspace=ws)
    ws.check()
    off = ws.ptr - ws.buf.data_ptr()
    header = ws.buf[off:off + 256].view(torch.int32)
    epoch, sparse_epoch = int(header[1]), int(header[11])
    assert (sparse_epoch == epoch - 1) == gathers
    exp = d_in.view(-1, GROUP_WORDS * 32)
    kept = torch.ones(len(exp), dtype=torch.bool, device="cuda")
    if every:
        kept[::every] = False
    exp = exp[kept][:, ::2].reshape(-1)  # bits 0, 2, 4, ...
    assert int(d_count.item()) == exp.numel()
    assert torch.equal(d_out[:exp.numel()], exp)
