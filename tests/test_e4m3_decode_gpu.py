"""Decode attention over e4m3 pages with f16 products: rows of q far from one, probabilities far below the largest, sinks and
splits, against the fp32 restatement."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,page,window,sinks,splits,q_scale", [
    (16, 1, 16, 0, False, 1, 1.0),          # sixteen heads of a group: every row of the product
    (8, 4, 32, 0, True, 1, 1e4),            # scores of hundreds: one key takes all
    (8, 4, 64, 0, True, 3, 1e-6),           # equal weights
    (5, 5, 16, 70, False, 2, 3.0),
])
def test_decode_over_e4m3_pages(Hq, Hkv, page, window, sinks, splits, q_scale):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(Hq * page)
    D, ctx = 128, [1, 15, 64, 65, 129, 700]
    need = [-(-c // page) for c in ctx]
    ids, at = torch.randperm(sum(need)).int(), 0
    table = torch.zeros(len(ctx), max(need), dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n], at = ids[at:at + n], at + n
    k, v = (torch.randn(sum(need), Hkv, page, D).to(torch.float8_e4m3fn) for _ in range(2))
    q = (torch.randn(len(ctx), Hq, D) * q_scale).bfloat16()
    q[0] = 0.0
    q[:, 0, 1:] = q[:, 0, 1:] * 2 ** -12    # one large element beside small ones
    s = torch.randn(Hq) if sinks else None
    kw = dict(window=window, num_splits=splits, max_ctx=max(ctx), kv_scale=(0.5, 3.0))
    cl = torch.tensor(ctx).int()
    got = cu.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), cl.cuda(), D ** -0.5, sinks=None if s is None else s.cuda(), **kw)
    cu.check_status(torch.device("cuda", 0))
    want = ref.attn_decode(q, k, v, table, cl, D ** -0.5, window=window, sinks=s, kv_scale=(0.5, 3.0))
    # one rounding of the output to bf16 (2^-9) on either side; probabilities are rounded to 2^-11
    assert float((got.cpu().float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("page,window,splits,byte", [(16, 0, 1, 0x7F), (32, 0, 3, 0xFF), (64, 70, 1, 0x7F), (16, 70, 9, 0xFF)])
def test_bytes_of_tokens_that_are_not_seen(page, window, splits, byte):
    """NaN bytes behind the contexts (a freed page keeps its contents) and ahead of the window change no bit."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(page + splits)
    Hq, Hkv, D, ctx = 8, 2, 128, [1, 15, 17, 64, 65, 130, 700]
    need = [-(-c // page) for c in ctx]
    ids, at = torch.randperm(sum(need)), 0
    table = torch.zeros(len(ctx), max(need), dtype=torch.int32)
    seen = torch.zeros(sum(need), page, dtype=torch.bool)
    for i, (n, c) in enumerate(zip(need, ctx)):
        mine, at = ids[at:at + n], at + n
        table[i, :n] = mine.int()
        rows = torch.zeros(n * page, dtype=torch.bool)
        rows[max(0, c - window) if window else 0:c] = True
        seen[mine] = rows.view(n, page)
    k, v = (torch.randn(sum(need), Hkv, page, D).to(torch.float8_e4m3fn).view(torch.uint8) for _ in range(2))
    q = torch.randn(len(ctx), Hq, D).bfloat16().cuda()
    out = []
    for fill in (0, byte):
        hidden = [t.masked_fill(~seen[:, None, :, None], fill).view(torch.float8_e4m3fn).cuda() for t in (k, v)]
        out.append(cu.attn_decode(q, *hidden, table.cuda(), torch.tensor(ctx).int().cuda(), D ** -0.5, window=window, num_splits=splits,
                                  max_ctx=max(ctx)))
    cu.check_status(torch.device("cuda", 0))
    assert bool(torch.isfinite(out[0].float()).all())
    assert torch.equal(*out)


@pytest.mark.parametrize("splits", [1, 3, 9])
def test_small_probabilities_keep_their_bits(splits):
    """Where the values of the keys that carry the softmax vanish, the others' make the output: here those of 2^-28.9."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(splits)
    Hkv, D, page, ctx = 2, 128, 16, 600
    nb = -(-ctx // page)
    table, cl = torch.randperm(nb).int().view(1, nb), torch.tensor([ctx]).int()
    k, v = torch.zeros(nb, Hkv, page, D), torch.randn(nb, Hkv, page, D)
    k[..., 0::2, 0], v[..., 1::2, :] = -0.9375, 0.0         # every other key scores -28.9 in powers of two, the rest 0
    k, v = k.to(torch.float8_e4m3fn), v.to(torch.float8_e4m3fn)
    q = torch.zeros(1, Hkv, D).bfloat16()
    q[..., 0] = 32.0
    scale = 28.9 / 30 * 0.6931471805599453
    got = cu.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), cl.cuda(), scale, max_ctx=ctx, num_splits=splits).cpu()
    want = ref.attn_decode(q, k, v, table, cl, scale)
    # outputs are rounded to bf16 (2^-8 at most, 2^-9 of a norm) on either side, probabilities to 2^-11
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -8
