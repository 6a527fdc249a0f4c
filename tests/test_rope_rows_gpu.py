"""Norm, rotation and cache write by vectors: head sizes, partial rotations on and off whole vectors, against the restatement."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,rot,Hq,Hkv", [(128, 128, 5, 1), (128, 32, 32, 8), (128, 16, 3, 3), (64, 64, 7, 1), (256, 64, 2, 1),
                                          (256, 256, 17, 2), (128, 24, 4, 2), (128, 0, 4, 2)])
@pytest.mark.parametrize("fp8", [False, True])
def test_norm_rotation_cache(D, rot, Hq, Hkv, fp8):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(D + rot)
    T, page, blocks = 37, 16, 5
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D).bfloat16()
    qn, kn = torch.randn(D).bfloat16(), torch.randn(D).bfloat16()
    cs = ref.build_cos_sin(300, rot, 1e4) if rot else None
    pos = torch.randint(0, 300, (T,)).int()
    slots = torch.randperm(blocks * page)[:T]
    slots[3] = -1
    kc = torch.zeros(blocks, Hkv, page, D, dtype=torch.float8_e4m3fn if fp8 else torch.bfloat16)
    kw = dict(norm_w_offset=1.0, kv_scale=(0.5, 2.0) if fp8 else (1.0, 1.0))
    a = [qkv.clone(), kc.clone(), kc.clone()]
    ref.qk_norm_rope_cache(a[0], qn, kn, cs, pos, slots, a[1], a[2], Hq, Hkv, D, rot, **kw)
    b = [qkv.cuda(), kc.cuda(), kc.cuda()]
    cu.qk_norm_rope_cache(b[0], qn.cuda(), kn.cuda(), None if cs is None else cs.cuda(), pos.cuda(), slots.cuda(), b[1], b[2], Hq, Hkv, D,
                          rot, **kw)
    cu.check_status(torch.device("cuda", 0))
    # a rounding to bf16 ahead of the rotation and one behind it; e4m3 keys: a step is 2^-3 of a value
    for x, y, lim in ((a[0][:, :Hq * D], b[0][:, :Hq * D], 2 ** -7), (a[1], b[1], 2 ** -4 if fp8 else 2 ** -7), (a[2], b[2], 0.0)):
        d = (x.float() - y.cpu().float()).norm() / x.float().norm()
        assert float(d) <= lim


@pytest.mark.parametrize("T", [1, 100, 197, 300, 700])      # a token's heads over three blocks, two and one
@pytest.mark.parametrize("D,Hq,Hkv", [(128, 32, 4), (64, 7, 30), (256, 9, 4)])
def test_blocks_per_token(T, D, Hq, Hkv):
    """However the heads of a token are shared out, every row comes out as in a batch of another size."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(T + D)
    n, page = 2000, 16
    qkv, pos = torch.randn(n, (Hq + 2 * Hkv) * D).bfloat16().cuda(), torch.randint(0, 300, (n,)).int().cuda()
    w, cs, slots = torch.randn(2, D).bfloat16().cuda(), ref.build_cos_sin(300, D, 1e4).cuda(), torch.randperm(n).cuda()
    out = []
    for rows in (n, T):
        x = [qkv[:rows].clone()] + [torch.zeros(n // page, Hkv, page, D, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        cu.qk_norm_rope_cache(x[0], w[0], w[1], cs, pos[:rows], slots[:rows], x[1], x[2], Hq, Hkv, D, D)
        at = slots[:T]
        out.append([x[0][:T]] + [c[at // page, :, at % page] for c in x[1:]])
    cu.check_status(torch.device("cuda", 0))
    assert all(torch.equal(a, b) for a, b in zip(*out))
