"""Prefill attention with two heads of a group per CTA (batches that fill the chip), against the fp32 restatement."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,page,kw", [
    (32, 8, 16, {}),
    (24, 12, 64, dict(window=200)),
    (64, 8, 32, dict(sinks=True)),
    (32, 4, 16, dict(window=150, keep_first=40)),
    (32, 8, 16, dict(softcap=20.0)),
    (32, 8, 16, dict(sigmoid=True)),
    (30, 10, 16, {}),                       # groups of three: one head per CTA
])
def test_prefill_pairs(Hq, Hkv, page, kw):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(Hq + page)
    D, kw = 128, dict(kw)
    # one token behind a cached prefix, ends on and off tiles of 128 rows and keys, a slice that starts inside a page
    seqs = [(1, 300), (128, 128), (129, 400), (257, 1000), (300, 300), (127, 131)]
    if kw.pop("sinks", False):
        kw["sinks"] = torch.randn(Hq)
    if kw.pop("sigmoid", False):
        kw["sigmoid_bias"] = torch.randn(Hq) - 3.0
    need = [-(-c // page) for _n, c in seqs]
    ids = torch.randperm(sum(need)).int()
    table, at = torch.zeros(len(seqs), max(need), dtype=torch.int32), 0
    for i, n in enumerate(need):
        table[i, :n], at = ids[at:at + n], at + n
    k, v = (torch.randn(sum(need), Hkv, page, D).bfloat16() for _ in range(2))
    T = sum(n for n, _c in seqs)
    q = (torch.randn(T, Hq, D) * 1.5).bfloat16()
    cu_q = torch.tensor([0] + [n for n, _c in seqs]).cumsum(0).int()
    ctx = torch.tensor([c for _n, c in seqs]).int()
    assert sum(-(-max(n for n, _c in seqs) // 128) for _ in seqs) * Hq // 2 >= 148
    to = lambda a: a.cuda() if isinstance(a, torch.Tensor) else a  # noqa: E731
    got = cu.attn_prefill(to(q), to(k), to(v), to(table), to(cu_q), to(ctx), max(n for n, _c in seqs), D ** -0.5,
                          **{n: to(a) for n, a in kw.items()}).cpu()
    cu.check_status(torch.device("cuda", 0))
    want = ref.attn_prefill(q, k, v, table, cu_q, ctx, max(n for n, _c in seqs), D ** -0.5, **kw)
    # probabilities and outputs are rounded to bf16 (2^-9 each)
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -7
