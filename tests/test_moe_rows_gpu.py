"""Rows of experts: taken into expert order, and put together again, at the edges of the kernels' parts."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (1, 8, 7168), (3, 2, 504), (7, 3, 520), (48, 2, 4096), (33, 8, 1032), (511, 8, 1024),
                                   (512, 8, 1024), (300, 5, 2880), (1030, 8, 264)])
def test_rows_in_expert_order(T, k, H):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(T)
    E = 16
    ids = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).int()
    ids[T // 2:, 0] = -1                     # pairs without an expert have no row
    plan = cu.moe_align(ids.cuda(), E)
    x = torch.randn(T, H).bfloat16()
    got, src = cu.moe_gather(x.cuda(), plan).cpu(), plan.src_tok.cpu().long()
    n = int(plan.offsets.cpu()[E])
    assert n == int((ids >= 0).sum())
    assert torch.equal(got[:n], x[src[:n]])


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (5, 2, 520), (9, 3, 2056), (741, 1, 256), (741, 5, 256), (1184, 4, 264), (1185, 8, 256),
                                   (1185, 2, 256)])
@pytest.mark.parametrize("base", [False, True])
def test_rows_put_together(T, k, H, base):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(T + k)
    E = 16
    ids = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).int()
    ids[::3, k - 1] = -1
    plan = cu.moe_align(ids.cuda(), E)
    y, w, b = torch.randn(T * k + 128, H).bfloat16(), torch.rand(T, k), torch.randn(T, H).bfloat16() if base else None
    got = cu.moe_combine(y.cuda(), plan, w.cuda(), None if b is None else b.cuda(), T).cpu()
    pos = plan.pos_of.cpu().long().view(T, k)
    want = torch.zeros(T, H) if b is None else b.float()
    for j in range(k):      # fp32 fused multiply-adds in the order of the experts: the same bits, however many rows are in flight
        more = (want.double() + y.double()[pos[:, j].clamp_min(0)] * w.double()[:, j:j + 1]).float()
        want = torch.where(pos[:, j:j + 1] >= 0, more, want)
    assert torch.equal(got, want.bfloat16())
