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
