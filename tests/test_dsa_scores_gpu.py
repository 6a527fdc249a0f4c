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
