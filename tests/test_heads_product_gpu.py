"""One or two rows: norm, product of the q, k and v heads, their norms, rotation and cache in one kernel."""

from ctypes import c_float, c_int, c_int64, c_void_p

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
P = c_void_p


def _fn():
    from parallax_b200.ops import _lib

    return _lib.bind("pxl_gemv_bf16_qkv", [P, P, c_float, c_float, P, P, P, P, P, P, P, P, P, P] + [c_int] * 7 + [c_int64, c_int, P, P])


@pytest.mark.parametrize("M,K", [(1, 8), (1, 256), (1, 1024), (1, 2568), (1, 4096), (2, 1024), (2, 5120)])
@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (16, 8), (14, 2)])
@pytest.mark.parametrize("normed,bias", [(True, False), (False, True)])
def test_heads(M, K, Hq, Hkv, normed, bias):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M + K + Hq)
    D, page, pages, eps = 128, 16, 6, 1e-6
    N = (Hq + 2 * Hkv) * D
    x, w_ln = torch.randn(M, K).bfloat16(), (1 + 0.1 * torch.randn(K)).bfloat16()
    w, b = (torch.randn(N, K) / K ** 0.5).bfloat16(), torch.randn(N).bfloat16() if bias else None
    qn, kn = ((1 + 0.1 * torch.randn(D)).bfloat16() for _ in range(2)) if normed else (None, None)
    angles = torch.rand(50, D // 2) * 6.28
    cos_sin = torch.cat([angles.cos(), angles.sin()], 1).float().contiguous()
    pos, slots = torch.tensor([7, 49][:M]).int(), torch.tensor([33, 80][:M]).long()

    xn = ref.rmsnorm(x, w_ln, eps)
    qkv = xn.float() @ w.float().t()
    qkv = (qkv + b.float() if bias else qkv).bfloat16()
    kc, vc = (torch.zeros(pages, Hkv, page, D).bfloat16() for _ in range(2))
    ref.qk_norm_rope_cache(qkv, qn, kn, cos_sin, pos, slots, kc, vc, Hq, Hkv, D, D, eps)

    g = lambda t: None if t is None else t.cuda()  # noqa: E731
    ptr = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    dev = torch.device("cuda", 0)
    a = [g(t) for t in (x, w_ln, w, b, qn, kn, cos_sin, pos, slots)]
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev)
    gk, gv = (torch.zeros(pages, Hkv, page, D, dtype=torch.bfloat16, device=dev) for _ in range(2))
    assert _fn()(ptr(a[0]), ptr(a[1]), eps, 0.0, ptr(a[2]), ptr(a[3]), ptr(out), ptr(a[4]), ptr(a[5]), ptr(a[6]), ptr(a[7]), ptr(a[8]),
                 ptr(gk), ptr(gv), M, K, Hq, Hkv, D, D, page, pages * page, 50, cu.status_tensor(dev).data_ptr(),
                 torch.cuda.current_stream().cuda_stream) == 0
    cu.check_status(dev)
    # the normed row, the product, the normed head and its rotation are rounded to bf16 (2^-9 each) on both sides
    for got, want in ((out[:, :Hq * D], qkv[:, :Hq * D]), (gk, kc), (gv, vc)):
        assert float((got.cpu().float() - want.float()).norm() / want.float().norm()) < 2 ** -7
    rows = torch.ones(pages * page, dtype=torch.bool)
    rows[slots] = False
    assert not gk.cpu().transpose(1, 2).reshape(-1, Hkv, D)[rows].any()


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_values_that_are_no_numbers(bad):
    """Value heads, and rows whose position is outside the table, are not rotated: a column that is no number leaves its other half alone."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(1)
    dev, D, Hq, Hkv, K, page = torch.device("cuda", 0), 128, 2, 1, 256, 16
    N = (Hq + 2 * Hkv) * D
    x, w_ln = torch.randn(1, K, device=dev).bfloat16(), torch.ones(K, device=dev).bfloat16()
    w, b = (torch.randn(N, K, device=dev) / K ** 0.5).bfloat16(), torch.randn(N, device=dev).bfloat16()
    marked = b.view(-1, D).clone()
    marked[:, 5] = bad
    cos_sin = torch.randn(8, D, device=dev)
    st = cu.status_tensor(dev).data_ptr()
    for pos, turned in ((3, True), (8, False)):
        p, slot = torch.tensor([pos], device=dev).int(), torch.tensor([1], device=dev).long()
        rows = []
        for bias in (marked, b):
            out = torch.zeros(1, N, dtype=torch.bfloat16, device=dev)
            k, v = (torch.zeros(1, Hkv, page, D, dtype=torch.bfloat16, device=dev) for _ in range(2))
            assert _fn()(x.data_ptr(), w_ln.data_ptr(), 1e-6, 0.0, w.data_ptr(), bias.data_ptr(), out.data_ptr(), None, None,
                         cos_sin.data_ptr(), p.data_ptr(), slot.data_ptr(), k.data_ptr(), v.data_ptr(), 1, K, Hq, Hkv, D, D, page, page, 8,
                         st, torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            if not turned:
                with pytest.raises(RuntimeError):
                    cu.check_status(dev)
            rows.append(torch.cat([out[0, :Hq * D].view(Hq, D), k[0, :, 1], v[0, :, 1]]))
        got, want = (t.cpu() for t in rows)
        away = torch.zeros(Hq + 2 * Hkv, D, dtype=torch.bool)
        away[:, 5] = True
        away[:Hq + Hkv, 5 + D // 2] = turned
        assert not got[away].isfinite().any()
        assert torch.equal(got[~away], want[~away])


def test_refused_and_reported():
    from parallax_b200.ops import _lib
    from parallax_b200.ops import cuda as cu

    takes = _lib.lib().pxl_gemv_bf16_qkv_takes
    assert takes(1, 1024, 16, 8, 128, 128) and takes(2, 1024, 16, 8, 128, 128)
    assert not any((takes(3, 1024, 16, 8, 128, 128), takes(1, 1024, 16, 8, 64, 64), takes(1, 1024, 16, 8, 128, 64), takes(1, 1020, 16, 8, 128, 128)))
    dev = torch.device("cuda", 0)
    x, w = torch.randn(1, 256, device=dev).bfloat16(), torch.randn(3 * 128, 256, device=dev).bfloat16()
    cs, out = torch.randn(4, 128, device=dev), torch.zeros(1, 3 * 128, device=dev, dtype=torch.bfloat16)
    k, v = (torch.zeros(1, 1, 16, 128, device=dev, dtype=torch.bfloat16) for _ in range(2))
    for pos, slot, ok in ((4, 0, False), (-1, 0, False), (0, 16, False), (0, -1, True)):
        p, s = torch.tensor([pos], device=dev).int(), torch.tensor([slot], device=dev).long()
        assert _fn()(x.data_ptr(), x.data_ptr(), 1e-6, 0.0, w.data_ptr(), None, out.data_ptr(), None, None, cs.data_ptr(), p.data_ptr(),
                     s.data_ptr(), k.data_ptr(), v.data_ptr(), 1, 256, 1, 1, 128, 128, 16, 16, 4, cu.status_tensor(dev).data_ptr(),
                     torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        if ok:
            cu.check_status(dev)
            continue
        with pytest.raises(RuntimeError):
            cu.check_status(dev)
    assert bool(k[0, 0, 0].any()) and not bool(k[0, 0, 1:].any())   # rows of bad positions are written unrotated, others have no place
