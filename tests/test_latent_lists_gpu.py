"""Latent attention over key lists (an indexer's choice) on the tensor cores, against the fp32 restatement."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,k,page,prompts,decode", [
    (128, 64, 16, [(5, 300)], [70, 129, 1]),         # whole tiles; a context shorter than the list
    (128, 200, 64, [(3, 256)], [201]),               # a last tile that is not full
    (8, 48, 8, [(40, 40), (2, 130)], [64]),          # fewer heads than rows: one token per tile; prompts from the start
    (192, 96, 128, [], [100, 500]),                  # two blocks of heads, pages longer than a tile
])
def test_latent_attention_over_lists(H, k, page, prompts, decode):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(H + k)
    L, R, scale = 512, 64, 192 ** -0.5
    ctx = [c for _n, c in prompts] + decode
    need = [-(-c // page) for c in ctx]
    blocks = torch.randperm(sum(need) + 3).int()
    table = torch.zeros(len(ctx), max(need), dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n], at = blocks[at:at + n], at + n
    cache = torch.randn(sum(need) + 3, 1, page, L + R).bfloat16()
    lens = [n for n, _c in prompts]
    for part in ("prompts", "decode"):
        if not (prompts if part == "prompts" else decode):
            continue
        first, seqs = (0, prompts) if part == "prompts" else (len(prompts), [(1, c) for c in decode])
        T = sum(n for n, _c in seqs)
        pos = torch.cat([torch.arange(c - n, c) for n, c in seqs])
        lists = torch.full((T, k), -1, dtype=torch.int32)
        for t in range(T):
            n = int(pos[t]) + 1
            if n > k:
                lists[t] = torch.randperm(n)[:k].int()
                if t % 2:       # an empty entry and a key that is not there yet
                    lists[t, 1], lists[t, 2] = -1, n + 1
        q = (torch.randn(T, H, L + R) * 0.5).bfloat16()
        cu_q = torch.tensor([0] + lens).cumsum(0).int() if part == "prompts" else None
        args = (cache, table[first:first + len(seqs)].contiguous(), cu_q, torch.tensor([c for _n, c in seqs]).int())
        kw = dict(max_q=max(n for n, _c in seqs), max_ctx=max(c for _n, c in seqs))
        want = ref.latent_attn(q, *args, scale, L, topk=lists, **kw)
        gpu = [a if a is None else a.cuda() for a in args]
        got = cu.latent_attn(q.cuda(), *gpu, scale, L, topk=lists.cuda(), **kw).cpu()
        cu.check_status(torch.device("cuda", 0))
        # probabilities and outputs are rounded to bf16 (2^-9 each)
        assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("H,page,prompts", [
    (128, 64, [(1, 130), (1, 64), (1, 1)]),     # decoding, one token per tile
    (24, 16, [(11, 75), (7, 7)]),               # five tokens and rows that are left over
    (192, 8, [(3, 70)]),                        # a second block of heads that fills half a tile
])
def test_wide_rows_with_a_part_of_the_query_in_tensor_memory(H, page, prompts):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(H)
    L, R = 512, 64
    need = [-(-c // page) for _n, c in prompts]
    table = torch.zeros(len(prompts), max(need), dtype=torch.int32)
    blocks, at = torch.randperm(sum(need)).int(), 0
    for i, n in enumerate(need):
        table[i, :n], at = blocks[at:at + n], at + n
    cache = torch.randn(sum(need), 1, page, L + R).bfloat16()
    q = (torch.randn(sum(n for n, _c in prompts), H, L + R) * 0.5).bfloat16()
    cu_q = torch.tensor([0] + [n for n, _c in prompts]).cumsum(0).int()
    args = (cache, table, cu_q, torch.tensor([c for _n, c in prompts]).int())
    kw = dict(max_q=max(n for n, _c in prompts), max_ctx=max(c for _n, c in prompts))
    want = ref.latent_attn(q, *args, 192 ** -0.5, L, **kw)
    got = cu.latent_attn(q.cuda(), *[a.cuda() for a in args], 192 ** -0.5, L, **kw).cpu()
    cu.check_status(torch.device("cuda", 0))
    # probabilities and outputs are rounded to bf16 (2^-9 each)
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("H,page,prompts,k,window", [
    (128, 64, [(1, 130), (1, 64), (1, 1)], 0, 0),       # decoding; a context that ends with its page
    (128, 16, [(1, 700), (1, 77)], 0, 100),             # keys ahead of the window, in the first tile's pages
    (24, 16, [(11, 75), (7, 7)], 0, 0),                 # tokens that share a tile: rows behind the last one's
    (192, 128, [(3, 70)], 0, 0),
    (16, 8, [(40, 130)], 48, 0),                        # lists, with entries that name no key
    (128, 64, [(1, 300), (1, 65)], 100, 0),             # a last tile of lists that is not full
])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_rows_that_are_not_seen(H, page, prompts, k, window, bad):
    """Cache rows behind a context, ahead of a window or off the lists that are no numbers change no bit."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(H + page)
    L, R, T = 512, 64, sum(n for n, _c in prompts)
    need = [-(-c // page) for _n, c in prompts]
    table = torch.zeros(len(prompts), max(need), dtype=torch.int32)
    blocks, at, t = torch.randperm(sum(need)), 0, 0
    seen = torch.zeros(sum(need), page, dtype=torch.bool)
    lists = torch.full((T, k), -1, dtype=torch.int32) if k else None
    for i, (n, (new, c)) in enumerate(zip(need, prompts)):
        mine, at = blocks[at:at + n], at + n
        table[i, :n] = mine.int()
        rows = torch.zeros(n * page, dtype=torch.bool)
        if k:       # a list per token out of the sequence's keys but the first one, short of a few entries
            for pos in range(c - new, c):
                keys = 1 + torch.randperm(pos)[:k]
                keys = keys if len(keys) < k else keys[:k - 3]
                lists[t, :len(keys)] = keys.int()
                rows[keys] = True
                t += 1
        else:
            rows[max(0, c - new - window + 1) if window else 0:c] = True
        seen[mine] = rows.view(n, page)
    cache = torch.randn(sum(need), 1, page, L + R).bfloat16()
    q = (torch.randn(T, H, L + R) * 0.5).bfloat16().cuda()
    cu_q = torch.tensor([0] + [n for n, _c in prompts]).cumsum(0).int().cuda()
    out = []
    for value in (0.0, bad):
        hidden = cache.masked_fill(~seen[:, None, :, None], value).cuda()
        out.append(cu.latent_attn(q, hidden, table.cuda(), cu_q, torch.tensor([c for _n, c in prompts]).int().cuda(), 192 ** -0.5, L,
                                  window=window, max_q=max(n for n, _c in prompts), max_ctx=max(c for _n, c in prompts),
                                  topk=None if lists is None else lists.cuda()))
    cu.check_status(torch.device("cuda", 0))
    assert bool(torch.isfinite(out[0].float()).all())
    assert torch.equal(*out)


@pytest.mark.parametrize("q_scale,bound", [(0.05, 2.3e-3), (1.0, 2.3e-3), (3.0, 1.95e-3)])
@pytest.mark.parametrize("lists", [False, True])
def test_error_against_64_bits(q_scale, bound, lists):
    """From flat to sharp distributions. Outputs are rounded to bf16 (1.66e-3 in the norm for random ones), and so are probabilities:
    another 1.4e-3 of the result as long as several keys count (2.2e-3 together), half of it or less once one key carries a row,
    whose rounding is above and below the line (1.8e-3)."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(3)
    B, H, L, R, page, ctx = 2, 128, 512, 64, 64, 2000
    nb, scale = -(-ctx // page), 192 ** -0.5
    cache, table = torch.randn(B * nb, 1, page, L + R).bfloat16().cuda(), torch.randperm(B * nb).int().view(B, nb).cuda()
    q, ctx_lens = (torch.randn(B, H, L + R) * q_scale).bfloat16().cuda(), torch.full((B,), ctx).int().cuda()
    topk = torch.stack([torch.randperm(ctx)[:1024] for _ in range(B)]).int().cuda() if lists else None
    got = cu.latent_attn(q, cache, table, None, ctx_lens, scale, L, max_ctx=ctx, topk=topk).double()
    cu.check_status(torch.device("cuda", 0))
    kv = cache.view(B * nb, page, L + R)[table.long()].view(B, nb * page, L + R)[:, :ctx].double()
    if lists:
        kv = torch.stack([k[t.long()] for k, t in zip(kv, topk)])
    p = torch.softmax(torch.einsum("bhd,bkd->bhk", q.double(), kv) * scale, -1)
    want = torch.einsum("bhk,bkd->bhd", p, kv[..., :L])
    err = float((got - want).norm() / want.norm())
    assert err < bound, err


@pytest.mark.parametrize("L,R,H,k,page,ctx", [
    (512, 32, 128, 130, 16, [400, 131]),    # a last column chunk that the rows do not fill; a last tile of two rows
    (480, 64, 128, 64, 64, [257, 64]),      # values that end inside a chunk; a context of one list's length
    (512, 8, 16, 200, 8, [1000]),           # few heads
    (448, 64, 128, 96, 16, [300]),          # eight column chunks
])
def test_lists_of_other_widths(L, R, H, k, page, ctx):
    """Rows off the lists are no numbers, also those that follow a listed row in memory."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(L + R)
    need = [-(-c // page) for c in ctx]
    table, at = torch.zeros(len(ctx), max(need), dtype=torch.int32), 0
    order = torch.randperm(sum(need)).int()
    for i, n in enumerate(need):
        table[i, :n], at = order[at:at + n], at + n
    cache = torch.randn(sum(need), 1, page, L + R).bfloat16()
    lists = torch.full((len(ctx), k), -1, dtype=torch.int32)
    for i, c in enumerate(ctx):
        if c > k:
            lists[i] = torch.randperm(c)[:k].int()
        keys = (lists[i] if c > k else torch.arange(c)).long()
        keep = torch.zeros(need[i] * page, dtype=torch.bool)
        keep[keys] = True
        rows = cache[table[i, :need[i]].long(), 0]
        rows.view(-1, L + R)[~keep] = float("nan")
        cache[table[i, :need[i]].long(), 0] = rows
    q = (torch.randn(len(ctx), H, L + R) * 0.5).bfloat16()
    lens, scale = torch.tensor(ctx).int(), 192 ** -0.5
    got = cu.latent_attn(q.cuda(), cache.cuda(), table.cuda(), None, lens.cuda(), scale, L, max_ctx=max(ctx), topk=lists.cuda()).cpu()
    cu.check_status(torch.device("cuda", 0))
    for i, c in enumerate(ctx):
        keys = (lists[i] if c > k else torch.arange(c)).long()
        rows = cache[table[i].long(), 0].reshape(-1, L + R)[keys].double()
        want = (q[i].double() @ rows.t() * scale).softmax(-1) @ rows[:, :L]
        # probabilities and outputs are rounded to bf16 (2^-9 each)
        assert float((got[i].double() - want).norm() / want.norm()) < 2 ** -7
