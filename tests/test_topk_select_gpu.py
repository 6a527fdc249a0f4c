"""Selection of the k best positions of a row: both ways of holding it, ties, lowest values."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [64, 2048, 8192, 8256, 20032])
@pytest.mark.parametrize("k", [1, 63, 64, 2048])
@pytest.mark.parametrize("values", ["normal", "ties", "equal", "infinite"])
def test_best_positions(width, k, values):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(width + k)
    ends = sorted({1, min(k, width), min(k + 1, width), width // 2 + 1, width - 1, width})
    s = torch.randn(len(ends), width)
    if values == "ties":
        s = (s * 2).round() / 2
    elif values == "equal":
        s = torch.full_like(s, -1.5)
    elif values == "infinite":
        s[:, ::3], s[:, 1::7] = float("-inf"), float("inf")
    pos = torch.tensor(ends).int() - 1
    got = cu.topk_select(s.cuda(), pos.cuda(), k).cpu()
    for row, n, chosen in zip(s, ends, got):
        if n <= k:
            assert bool((chosen == -1).all())
            continue
        assert chosen.unique().numel() == k and int(chosen.min()) >= 0 and int(chosen.max()) < n
        assert torch.equal(row[chosen.long()].sort().values, row[:n].topk(k).values.sort().values)
