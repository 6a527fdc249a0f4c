"""Decode attention in splits: added inside clusters where all of them are on the chip at once, through the workspace otherwise."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,splits,kernels", [(1, 8, 1), (2, 9, 2), (74, 2, 1), (80, 2, 2), (40, 5, 2)])
@pytest.mark.parametrize("fp8,kw", [(False, {}), (False, dict(softcap=20.0)), (False, dict(sigmoid=True)), (False, dict(sinks=True)),
                                    (True, dict(sinks=True))])
def test_splits(B, splits, kernels, fp8, kw):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(B + splits)
    Hq, Hkv, D, page, kw = 8, 2, 128, 16, dict(kw)
    ctx = torch.tensor([1 + 37 * i % 640 for i in range(B)]).int()      # some splits have no keys
    if kw.pop("sinks", False):
        kw["sinks"] = torch.randn(Hq)
    if kw.pop("sigmoid", False):
        kw["sigmoid_bias"] = torch.randn(Hq) - 3.0
    table = torch.randperm(B * 40).int().view(B, 40)
    k, v = (torch.randn(B * 40, Hkv, page, D).to(torch.float8_e4m3fn if fp8 else torch.bfloat16) for _ in range(2))
    q = torch.randn(B, Hq, D).bfloat16()
    to = lambda a: a.cuda() if isinstance(a, torch.Tensor) else a  # noqa: E731
    before = cu.launch_count
    got = cu.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), ctx.cuda(), D ** -0.5, max_ctx=640, num_splits=splits,
                         **{n: to(a) for n, a in kw.items()})
    assert cu.launch_count - before == kernels
    cu.check_status(torch.device("cuda", 0))
    want = ref.attn_decode(q, k, v, table, ctx, D ** -0.5, **kw)
    # probabilities and outputs are rounded to bf16 (2^-9 each)
    assert float((got.cpu().float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("D,page", [(128, 16), (128, 8), (64, 16)])
@pytest.mark.parametrize("B,most", [(1, 64), (1, 65), (1, 777), (9, 129), (75, 640)])
def test_chosen_splits(D, page, B, most):
    from parallax_b200.ops import _lib
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(B + most)
    Hq, Hkv, blocks = 8, 2, -(-most // page)
    s = _lib.lib().pxl_attn_decode_splits(B, Hq, Hkv, D, page, 0, most)
    tiles = -(-most // 64)
    assert 1 <= s <= 64 and (s <= tiles or B * Hkv * s >= 4 * torch.cuda.get_device_properties(0).multi_processor_count)
    ctx = torch.tensor([most - 41 * i % most for i in range(B)]).int()
    table = torch.randperm(B * blocks).int().view(B, blocks)
    k, v = (torch.randn(B * blocks, Hkv, page, D).bfloat16() for _ in range(2))
    q = torch.randn(B, Hq, D).bfloat16()
    got = cu.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), ctx.cuda(), D ** -0.5, max_ctx=most)
    cu.check_status(torch.device("cuda", 0))
    want = ref.attn_decode(q, k, v, table, ctx, D ** -0.5)
    # probabilities and outputs are rounded to bf16 (2^-9 each)
    assert float((got.cpu().float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("lens", ["one tile", "edges", "ragged", "long"])
@pytest.mark.parametrize("Hq,Hkv,page", [(8, 2, 16), (8, 1, 32), (21, 7, 64)])
@pytest.mark.parametrize("fp8,kw", [(False, {}), (False, dict(softcap=20.0)), (False, dict(sigmoid=True)), (False, dict(sinks=True)),
                                    (False, dict(window=130, keep_first=70)), (True, dict(sinks=True)), (True, dict(window=96))])
def test_even_tiles(lens, Hq, Hkv, page, fp8, kw):
    """Splits that give two places per CTA: the tiles of all pairs are dealt out evenly."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(7)
    kw, D = dict(kw), 128
    ctx = {"one tile": [1 + i % 64 for i in range(70)], "edges": [1, 63, 64, 65, 127, 128, 129, 640, 0, 5] * 7,
           "ragged": [1 + i * i * 37 % 900 for i in range(75)], "long": [3, 5000, 1, 64, 2 * 64, 4097]}[lens]
    B, most = len(ctx), max(ctx)
    splits = -(-4 * torch.cuda.get_device_properties(0).multi_processor_count // (B * Hkv))
    if splits < 2:
        splits = 2
    if kw.pop("sinks", False):
        kw["sinks"] = torch.randn(Hq)
    if kw.pop("sigmoid", False):
        kw["sigmoid_bias"] = torch.randn(Hq) - 3.0
    blocks = -(-most // page)
    table = torch.randperm(B * blocks).int().view(B, blocks)
    k, v = (torch.randn(B * blocks, Hkv, page, D).to(torch.float8_e4m3fn if fp8 else torch.bfloat16) for _ in range(2))
    q = torch.randn(B, Hq, D).bfloat16()
    to = lambda a: a.cuda() if isinstance(a, torch.Tensor) else a  # noqa: E731
    lens_t = torch.tensor(ctx).int()
    got = cu.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), lens_t.cuda(), D ** -0.5, max_ctx=most, num_splits=splits,
                         **{n: to(a) for n, a in kw.items()})
    cu.check_status(torch.device("cuda", 0))
    keep = lens_t > 0
    want = ref.attn_decode(q[keep], k, v, table[keep], lens_t[keep], D ** -0.5, **kw)
    # probabilities and outputs are rounded to bf16 (2^-9 each)
    assert float((got.cpu().float()[keep] - want.float()).norm() / want.float().norm()) < 2 ** -7
    assert bool((got.cpu()[~keep] == 0).all())
