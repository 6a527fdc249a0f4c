"""Indexer scores of groups of tokens that cross sequences, against the fp32 restatement."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hi,page", [(64, 16), (24, 64), (3, 8)])
def test_scores_of_ragged_prompts(Hi, page):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(Hi)
    # ends of groups, of sequences and of the 128-key tiles in all orders; a slice behind a cached prefix
    seqs = [(130, 130), (1, 257), (5, 700), (251, 640), (40, 129)]
    need = [-(-c // page) for _n, c in seqs]
    ids, at = torch.randperm(sum(need)).int(), 0
    table = torch.zeros(len(seqs), max(need), dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n], at = ids[at:at + n], at + n
    T, max_ctx = sum(n for n, _c in seqs), max(c for _n, c in seqs)
    cache = torch.randn(sum(need), 1, page, 128).bfloat16()
    q, w = torch.randn(T, Hi, 128).bfloat16(), torch.randn(T, Hi)
    pos = torch.cat([torch.arange(c - n, c) for n, c in seqs]).int()
    cu_q = torch.tensor([0] + [n for n, _c in seqs]).cumsum(0).int()
    got = cu.dsa_index_scores(*[t.cuda() for t in (q, w, cache, table, cu_q, pos)], max_ctx).cpu()
    want = ref.dsa_index_scores(q, w, cache, table, cu_q, pos, max_ctx)
    seen = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), seen)
    # bf16 products are exact in fp32; sums of 128 and of Hi terms in another order
    assert float((got[seen] - want[seen]).norm() / want[seen].norm()) < 1e-5


@pytest.mark.parametrize("max_ctx,width", [(40, 64), (65, 128), (129, 192), (320, 320)])
def test_columns_beyond_the_keys_stay(max_ctx, width):
    """Rows of scores inside a wider buffer: columns up to the next multiple of 64 are written, those behind are someone else's."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(max_ctx)
    T, Hi, page = 3, 8, 16
    q, w = torch.randn(T, Hi, 128).bfloat16().cuda(), torch.randn(T, Hi).cuda()
    cache, table = torch.randn(20, 1, page, 128).bfloat16().cuda(), torch.arange(20).int().view(1, 20).cuda()
    pos, cu_q = torch.arange(max_ctx - T, max_ctx).int().cuda(), torch.tensor([0, T]).int().cuda()
    wide = torch.full((T, 512), 7.0, device="cuda")
    code = cu._lib.lib().pxl_dsa_index_scores(q.data_ptr(), w.data_ptr(), cache.data_ptr(), table.data_ptr(), cu_q.data_ptr(),
                                              pos.data_ptr(), wide.data_ptr(), 512, T, 1, Hi, 128, 20, page, max_ctx,
                                              torch.cuda.current_stream().cuda_stream)
    assert code == 0
    assert torch.equal(wide[:, :width], cu.dsa_index_scores(q, w, cache, table, cu_q, pos, max_ctx))
    assert bool((wide[:, width:] == 7.0).all())


def test_tokens_in_any_order():
    """Positions of a sequence that do not rise from token to token."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(9)
    lens, ctx, page, Hi = [70, 200], [300, 513], 16, 16
    table = torch.randperm(2 * 33).int().view(2, 33)
    cache = torch.randn(66, 1, page, 128).bfloat16()
    pos = torch.cat([c - 1 - torch.randperm(n) for n, c in zip(lens, ctx)]).int()
    q, w = torch.randn(sum(lens), Hi, 128).bfloat16(), torch.randn(sum(lens), Hi)
    cu_q = torch.tensor([0, 70, 270]).int()
    got = cu.dsa_index_scores(*[t.cuda() for t in (q, w, cache, table, cu_q, pos)], max(ctx)).cpu()
    want = ref.dsa_index_scores(q, w, cache, table, cu_q, pos, max(ctx))
    seen = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), seen)
    assert float((got[seen] - want[seen]).norm() / want[seen].norm()) < 1e-5      # fp32 sums in another order


@pytest.mark.parametrize("Hi", [32, 64])
@pytest.mark.parametrize("lens,ctx,shuffled", [([2], [2], False), ([1, 130, 3], [300, 130, 512], False), ([257], [257], True),
                                               ([600], [1700], False), ([40, 1, 90], [255, 256, 1030], True)])
def test_scores_of_32_and_64_heads(Hi, lens, ctx, shuffled):
    """256 keys per CTA and tiles of 128 / heads tokens: ends of sequences, groups and tiles, keys nobody sees."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(sum(lens) + Hi)
    page = 16
    need = [-(-c // page) for c in ctx]
    ids, at = torch.randperm(sum(need)).int(), 0
    table = torch.full((len(lens), max(need)), -1, dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n], at = ids[at:at + n], at + n
    T, most = sum(lens), max(ctx)
    pos = torch.cat([(torch.arange(c - n, c)[torch.randperm(n)] if shuffled else torch.arange(c - n, c)) for n, c in zip(lens, ctx)]).int()
    cache = torch.randn(sum(need), 1, page, 128).bfloat16()
    q, w = torch.randn(T, Hi, 128).bfloat16(), torch.randn(T, Hi)
    cu_q = torch.tensor([0] + lens).cumsum(0).int()
    got = cu.dsa_index_scores(*[t.cuda() for t in (q, w, cache, table, cu_q, pos)], most).cpu()
    cu.check_status(torch.device("cuda", 0))
    want = ref.dsa_index_scores(q, w, cache, table.clamp(min=0), cu_q, pos, most)
    seen = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), seen)
    # bf16 products are exact in fp32; sums of 128 and of Hi terms in another order
    assert float((got[seen] - want[seen]).norm() / want[seen].norm()) < 1e-5


@pytest.mark.parametrize("Hi,prompt", [(64, True), (32, True), (24, True), (64, False)])
@pytest.mark.parametrize("entry", [-1, 20, 1 << 30])
def test_entries_outside_the_cache(Hi, prompt, entry):
    """A table entry that is no block of the cache, where a token sees it: reported, and block 0 in its place."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(Hi)
    dev, page, pages, T = torch.device("cuda", 0), 16, 20, 40 if prompt else 3
    B, ctx = (1, 310) if prompt else (T, 310)
    table = torch.arange(pages).int().repeat(B, 1)
    bad = table.clone()
    bad[0, 7], table[0, 7] = entry, 0
    cache = torch.randn(pages, 1, page, 128).bfloat16()
    q, w = torch.randn(T, Hi, 128).bfloat16(), torch.randn(T, Hi)
    pos = (torch.arange(ctx - T, ctx) if prompt else torch.full((T,), ctx - 1)).int()
    cu_q = torch.tensor([0, T]).int().cuda() if prompt else None
    a = [t.cuda() for t in (q, w, cache)]
    want = cu.dsa_index_scores(*a, table.cuda(), cu_q, pos.cuda(), ctx)
    cu.check_status(dev)
    got = cu.dsa_index_scores(*a, bad.cuda(), cu_q, pos.cuda(), ctx)
    with pytest.raises(RuntimeError):
        cu.check_status(dev)
    assert torch.equal(got, want)
    if entry < 0:       # a position behind the table
        got = cu.dsa_index_scores(*a, table.cuda()[:, :7].contiguous(), cu_q, pos.cuda(), ctx)
        with pytest.raises(RuntimeError):
            cu.check_status(dev)
        assert bool(torch.isfinite(got[:, :ctx - T]).all())


@pytest.mark.parametrize("Hi,each", [(64, 1), (64, 2), (32, 3), (32, 4)])
def test_many_short_prompts(Hi, each):
    """Fewer tokens per prompt than a tile of the tensor cores' kernel (128 / heads), and as many."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(each)
    page, ctx, B = 16, 300, 20
    pages = -(-ctx // page)
    table, cache = torch.randperm(B * pages).int().view(B, pages), torch.randn(B * pages, 1, page, 128).bfloat16()
    T = B * each
    pos = torch.cat([torch.arange(ctx - 7 * i - each, ctx - 7 * i) for i in range(B)]).int()
    q, w, cu_q = torch.randn(T, Hi, 128).bfloat16(), torch.randn(T, Hi), (torch.arange(B + 1) * each).int()
    got = cu.dsa_index_scores(*[t.cuda() for t in (q, w, cache, table, cu_q, pos)], ctx).cpu()
    cu.check_status(torch.device("cuda", 0))
    want = ref.dsa_index_scores(q, w, cache, table, cu_q, pos, ctx)
    seen = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), seen)
    assert float((got[seen] - want[seen]).norm() / want[seen].norm()) < 1e-5      # fp32 sums in another order
