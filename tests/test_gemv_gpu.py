"""Products of a handful of rows without tensor cores, and with the RMS norm inside, against the fp32 restatement."""

import ctypes

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.float().cpu() - b.float().cpu()).norm() / b.float().cpu().norm())


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 264), (3600, 512), (7296, 2056)])       # 1, 2 and 4 rows of W per warp; ends of K
def test_few_rows(M, N, K):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M * N + K)
    x, w = torch.randn(M, K + 8).bfloat16()[:, :K], (torch.randn(N, K) * 0.05).bfloat16()
    b, r = torch.randn(N).bfloat16(), torch.randn(M, N).bfloat16()
    g = lambda t: t.cuda()  # noqa: E731
    want = x.float() @ w.float().t()
    # fp32 sums; one rounding to bf16 (2^-9) behind them
    assert _rel(cu.linear(g(x), g(w)), want) < 2 ** -8
    assert _rel(cu.linear(g(x), g(w), bias=g(b)), want + b.float()) < 2 ** -8
    assert _rel(cu.linear(g(x), g(w), bias=g(b), residual=g(r)), want + b.float() + r.float()) < 2 ** -8
    assert _rel(cu.linear(g(x), g(w), epi=ref.EPI_F32), want) < 1e-5


@pytest.mark.parametrize("M", [1, 2, 3, 5])
@pytest.mark.parametrize("N,K", [(128, 72), (4096, 1024), (15360, 256)])
def test_few_rows_gated(M, N, K):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M + N)
    x = torch.randn(M, K).bfloat16().cuda()
    wg, wu = ((torch.randn(N // 2, K) * 0.1).bfloat16().cuda() for _ in range(2))
    want = torch.nn.functional.silu(x.float() @ wg.float().t()) * (x.float() @ wu.float().t())
    assert _rel(cu.linear(x, ref.interleave_gate_up(wg, wu), epi=ref.EPI_SILU_MUL), want) < 2 ** -8


@pytest.mark.parametrize("M,N,K,glu", [(1, 264, 1024, False), (2, 5120, 520, False), (1, 6144, 1024, True), (2, 256, 4096, True)])
def test_norm_inside(M, N, K, glu):
    from parallax_b200.ops import cuda as cu

    c = ctypes
    fn = cu._lib.bind("pxl_gemv_bf16_norm", [c.c_void_p] * 2 + [c.c_float] * 2 + [c.c_void_p] * 3 + [c.c_int] * 7 + [c.c_void_p])
    torch.manual_seed(N)
    x, nw = torch.randn(M, K).bfloat16().cuda() * 3, (torch.randn(K) * 0.2).bfloat16().cuda()
    w = (torch.randn(N, K) * 0.05).bfloat16().cuda()
    out = torch.empty(M, N // 2 if glu else N, dtype=torch.bfloat16, device="cuda")
    args = (x.data_ptr(), nw.data_ptr(), 1e-6, 1.0, w.data_ptr(), out.data_ptr(), None, M, N, K, K, K, out.shape[1])
    assert fn(*args, ref.EPI_SILU_MUL if glu else 0, torch.cuda.current_stream().cuda_stream) == 0
    xn = ref.rmsnorm(x, nw, 1e-6, w_offset=1.0)
    want = ref.linear(xn, w, epi=ref.EPI_SILU_MUL if glu else 0)
    assert _rel(out, want) < 2 ** -7        # (the reference rounds to bf16, too; a normed value may round the other way)
