"""Block tables made by a kernel of a launch chain, read by the decode attention behind it."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_selected_blocks_in_a_chain():
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(3)
    dev, T, Hq, Hkv, D, page, block, topk, ctx = torch.device("cuda", 0), 8, 8, 2, 128, 16, 64, 4, 1000
    pages = -(-ctx // page)
    table = torch.randperm(T * pages).int().view(T, pages).to(dev)
    k, v = (torch.randn(T * pages, Hkv, page, D, device=dev).bfloat16() for _ in range(2))
    q, w = torch.randn(T, Hq, D, device=dev).bfloat16(), torch.ones(D, device=dev).bfloat16()
    pos = torch.full((T,), ctx - 1, device=dev, dtype=torch.int32)
    scores = [torch.randn(T, -(-ctx // block), device=dev) for _ in range(20)]

    def step(s):
        cu.rmsnorm(q.view(-1, D), w, 1e-6)
        vt, vctx = cu.msa_select(s, pos, table, None, page, block, topk, 1, 1)
        return cu.attn_decode(q, k, v, vt, vctx, D ** -0.5, max_ctx=topk * block)

    want = [step(s) for s in scores]
    torch.cuda.synchronize()
    with cu.launch_chain():
        got = [step(s) for s in scores]
    cu.check_status(dev)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
