"""Long columns of which everything, or all but a few elements, is selected, through the 3-pass form: the
writeout leaves some of its warps idle there, by the share that is selected. Bit for bit against the
input. Needs a B200."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("dropped", [0, 1, 1 << 12, 1 << 18])
def test_nearly_all_selected(cuda, w, dropped):
    import torch
    import gpu_compressstore2_b200 as cs

    n = (8 * 148 * 3 * 8 * 4096 + 5000) // w + 77  # 8 items of 4 KB for every warp and more
    dt = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[w]
    g = torch.Generator(device="cuda")
    g.manual_seed(w)
    x = torch.randint(0, 1 << 7, (n,), dtype=dt, device="cuda", generator=g)
    keep = torch.ones((n + 127) // 128 * 128, dtype=torch.bool, device="cuda")
    if dropped:
        keep[torch.randint(0, n, (dropped,), device="cuda", generator=g)] = False
    bits = keep.view(-1, 8).to(torch.uint8)
    mask = sum(bits[:, b] << b for b in range(8)).to(torch.uint8).view(torch.int32)
    out = torch.full((n + 64,), 77, dtype=dt, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    cs.compressstore(x, mask, out, n, count, algo=cs.ALGO_3PASS)
    exp = x[keep[:n]]
    assert int(count.item()) == exp.numel()
    assert torch.equal(out[:exp.numel()], exp)
    assert bool((out[exp.numel():] == 77).all())
