"""The form that a plan takes by its columns (one launch where they are all short, or of one width and 16 or
28 to 80 MB, two and more otherwise), and long plans whose writeouts leave warps idle. Every column against torch's
own indexing. Needs a B200."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _plan(specs, seed=1):
    """Columns (n, element bytes, selected share) and a plan over them."""
    import torch
    import gpu_compressstore2_b200 as cs

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    counts = torch.zeros(len(specs), dtype=torch.int64, device="cuda")
    cols, keeps = [], []
    for i, (n, w, p) in enumerate(specs):
        dt = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[w]
        keep = torch.zeros((n + 127) // 128 * 128, dtype=torch.bool, device="cuda")
        keep[:n] = torch.rand(n, device="cuda", generator=g) < p if p < 1 else True
        bits = keep.view(-1, 8).to(torch.uint8)
        mask = sum(bits[:, b] << b for b in range(8)).to(torch.uint8).view(torch.int32)
        x = torch.randint(0, 1 << 7, (n,), dtype=dt, device="cuda", generator=g)
        cols.append((x, mask, torch.full((n + 16,), 77, dtype=dt, device="cuda"), n, counts[i:i + 1]))
        keeps.append(keep[:n])
    torch.cuda.synchronize()
    return cs.Batch(cols), cols, keeps, counts


def _check(specs, launches):
    import torch

    plan, cols, keeps, counts = _plan(specs)
    assert plan.launches_per_run == launches
    for _ in range(2):
        plan.run()
        plan.check()
        for (x, _, out, n, _), keep, k in zip(cols, keeps, counts.tolist()):
            exp = x[keep]
            assert k == exp.numel()
            assert torch.equal(out[:k], exp)
            assert bool((out[k:] == 77).all())
            out.fill_(77)
    plan.close()


SHORT, MIDDLE = 1 << 14, 10 << 20  # elements, bytes


@pytest.mark.parametrize("specs,launches", [
    ([(SHORT, 4, 0.5)], 1),
    ([(SHORT + 1, 4, 0.5)], 2),
    ([(100 + i, 8, 0.9) for i in range(40)], 1),
    ([(SHORT - i, 2, 0.3) for i in range(8)], 1),
    ([(SHORT - i, 2, 0.3) for i in range(9)], 2),
    ([(SHORT, 1, 0.5)], 2),
    ([(SHORT, 4, 0.5), (SHORT, 8, 0.5)], 3),
    ([(SHORT, 4, 0.5), (0, 8, 0.5)], 1),
    ([(SHORT - i, 2, 0.3) for i in range(129)], 1),
    ([(7 << 20, 4, 0.6)], 1),
    ([((7 << 20) - 1, 4, 0.6)], 2),
    ([(2 << 20, 8, 0.6)], 1),
    ([((2 << 20) - 1, 8, 0.6)], 2),
    ([(MIDDLE // 4 + i, 4, 0.1) for i in range(4)], 1),
    ([(MIDDLE // 4 + i, 4, 0.01) for i in range(4)], 2),
    ([(MIDDLE // 8 + i, 8, 0.1) for i in range(4)], 2),
    ([(MIDDLE // 8 + i, 8, 0.5) for i in range(8)], 2),
    ([(MIDDLE // 8 - i, 8, 0.5) for i in range(8)], 1),
    ([(MIDDLE // 2 - i, 2, 0.8) for i in range(5)], 1),
    ([(MIDDLE - i, 1, 0.8) for i in range(5)], 2),
])
def test_form_by_columns(cuda, specs, launches):
    _check(specs, launches)


@pytest.mark.parametrize("w,share", [(8, 0.76), (8, 1), (4, 0.9), (4, 1)])
def test_long_plans_mostly_selected(cuda, w, share):
    """More than 8 items of 4 KB for every warp, in columns of odd lengths."""
    n = 148 * 3 * 8 * 8 * 4096 // w // 3 + 1001
    _check([(n + i, w, share) for i in range(4)] + [(5000, w, 0.01)], 2)


@pytest.mark.parametrize("share", [0.74, 0.76, 1])
def test_idle_warps_of_plans(cuda, share):
    """512 MB and more of 8-byte columns, and a narrower and a short one beside them."""
    _check([((64 << 20) // 3 + 1001 + i, 8, share) for i in range(3)] + [(5000, 8, 0.01)], 2)
    _check([((64 << 20) // 3 + 1001 + i, 8, share) for i in range(3)] + [(70001, 4, 0.9)], 3)
