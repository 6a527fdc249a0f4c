"""Decode attention of rows of unlike lengths: one long row beside short ones is not left to a CTA or two."""

import numpy as np
import pytest
import torch

from parallax_b200.engine.batch import BatchBuilder
from parallax_b200.ops import reference as ref


def test_keys_of_all_rows():
    table = np.zeros((3, 4), dtype=np.int32)
    fb = BatchBuilder(torch.device("cpu"), 8, 4, 16).build(
        None, np.array([4, 60, 0], dtype=np.int32), np.zeros(3, dtype=np.int64), [], [], None, np.array([5, 61, 1], dtype=np.int32),
        table, np.arange(3, dtype=np.int32))
    assert (fb.d_max_ctx, fb.d_total_ctx) == (61, 67)


@pytest.mark.gpu
@pytest.mark.parametrize("D,fp8,G", [(128, 0, 4), (128, 1, 4), (64, 0, 8)])
@pytest.mark.parametrize("B,Hkv", [(14, 8), (32, 8), (64, 4), (200, 1)])
def test_long_row_beside_short_ones(B, Hkv, D, fp8, G):
    from parallax_b200.ops import _lib

    most, total, chip = 32768, 32768 + (B - 1) * 1000, 2 * torch.cuda.get_device_properties(0).multi_processor_count
    s = _lib.lib().pxl_attn_decode_splits_of(B, Hkv * G, Hkv, D, 64, fp8, most, total)
    # at least half as many again as places for CTAs, by which the long row's chain of 512 tiles is a third of what one split leaves
    assert s >= 3 or B * Hkv * s >= 2 * chip
    for keys in (0, B * most, 1 << 40):      # not known, or all rows as long as the longest
        assert _lib.lib().pxl_attn_decode_splits_of(B, Hkv * G, Hkv, D, 64, fp8, most, keys) == \
            _lib.lib().pxl_attn_decode_splits(B, Hkv * G, Hkv, D, 64, fp8, most)


@pytest.mark.gpu
@pytest.mark.parametrize("D,fp8,page", [(128, False, 16), (128, True, 64), (64, False, 16), (128, False, 8)])
@pytest.mark.parametrize("B,Hkv,most", [(3, 1, 3000), (20, 2, 5000), (40, 8, 2500), (150, 2, 1900)])
def test_uneven_rows(B, Hkv, most, D, fp8, page):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(B)
    ctx = torch.tensor([1 + 37 * i % 150 for i in range(B)]).int()
    ctx[B // 2] = most
    pages = [-(-int(c) // page) for c in ctx]
    table, order, at = torch.zeros(B, max(pages)).int(), torch.randperm(sum(pages)).int(), 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    k, v = (torch.randn(sum(pages), Hkv, page, D).to(torch.float8_e4m3fn if fp8 else torch.bfloat16) for _ in range(2))
    q = torch.randn(B, Hkv * 4, D).bfloat16()
    got = cu.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), ctx.cuda(), D ** -0.5, max_ctx=most, total_ctx=int(ctx.sum()))
    cu.check_status(torch.device("cuda", 0))
    want = ref.attn_decode(q, k, v, table, ctx, D ** -0.5, total_ctx=int(ctx.sum()))
    err = (got.cpu().float() - want.float()).flatten(1).norm(dim=1) / want.float().flatten(1).norm(dim=1)
    # probabilities and outputs are rounded to bf16 (2^-9 each), row by row
    assert float(err.max()) < 2 ** -7
