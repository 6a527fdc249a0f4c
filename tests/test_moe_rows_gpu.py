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
