"""Causal convolution of decoded tokens by pairs of channels against the form that takes a channel per thread: the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,C,bias", [([1] * 5, 8192, False), ([1, 3, 1], 258, True), ([2], 2, False)])
def test_pairs_of_channels(lens, C, bias):
    from parallax_b200.ops import cuda as cu

    g = torch.Generator(device="cuda").manual_seed(C)
    T, B = sum(lens), len(lens)

    def rnd(*shape):
        return torch.randn(*shape, device="cuda", dtype=torch.bfloat16, generator=g)

    x, w, b, s = rnd(T, C + 6), rnd(C, 4), rnd(C) if bias else None, rnd(B + 2, C, 3)
    cu_q = torch.tensor([0] + lens).cumsum(0).int().cuda()
    slots = torch.randperm(B + 2, generator=torch.Generator().manual_seed(1))[:B].int().cuda()
    pos = torch.cat([torch.arange(p, p + n) for p, n in zip([7, 0, 300, 4, 0], lens)]).int().cuda()
    odd = torch.zeros(w.numel() + 1, device="cuda", dtype=torch.bfloat16)[1:].view(C, 4).copy_(w)      # off the 16 bytes: the other form
    res = []
    for weights in (w, odd):
        state = s.clone()
        res.append((cu.causal_conv1d_silu(x[:, :C], weights, b, state, cu_q, slots, pos), state))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    win = torch.where((pos[cu_q[:-1].long()] == 0)[:, None, None], 0.0, s[slots.long()].double())
    for i, n in enumerate(lens):
        a = int(cu_q[i])
        u = torch.cat([win[i].t(), x[a:a + n, :C].double()], 0)
        y = (u.unfold(0, 4, 1) * w.double()).sum(-1) + (0 if b is None else b.double())
        want = torch.nn.functional.silu(y)
        assert float((res[0][0][a:a + n].double() - want).norm() / want.norm()) < 2 ** -7
        assert torch.equal(res[0][1][int(slots[i])].double(), u[-3:].t())
