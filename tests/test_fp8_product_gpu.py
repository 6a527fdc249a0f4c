"""Block-scaled fp8 product and the quantisation of its rows, against the fp32 restatement."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (130, 256, 384), (64, 128, 512), (257, 384, 1152)])
def test_fp8_product_and_row_quantisation(M, N, K):
    """Numbers of K blocks that the groups of four scales do and do not divide; rows at an odd stride."""
    from parallax_b200.loader.quant import quantize_fp8_block
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M + K)
    x = torch.randn(M, K + 3).bfloat16()[:, :K]
    w, s = quantize_fp8_block(torch.randn(N, K) * 0.05, (64, 128))
    xq, xs = ref.quant_fp8_rows(x)
    gq, gs = cu.quant_fp8_rows(x.cuda())
    assert torch.allclose(gs.cpu(), xs, rtol=1e-6)
    # quotients that differ in their last fp32 bit may round to neighbouring codes: a step is at most 2^-3 of a value, and
    # values below 2^-6 share its step
    a, b = gq.cpu().float(), xq.float()
    assert bool(((a - b).abs() <= b.abs().clamp_min(2.0 ** -6) * 2.0 ** -3).all())
    got, want = cu.linear_fp8(x.cuda(), w.cuda(), s.cuda()).cpu(), ref.linear_fp8(x, w, s)
    cu.check_status(torch.device("cuda", 0))
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("M,N,K", [(1, 128, 2048), (64, 256, 4096), (100, 128, 2304), (130, 256, 2176)])
@pytest.mark.parametrize("epi", ["plain", "residual", "glu"])
def test_fp8_product_split_over_a_cluster(M, N, K, epi):
    """Few output tiles: K in ranges (also of unequal lengths), the rows of a tile shared out over the CTAs that add them."""
    from parallax_b200.loader.quant import quantize_fp8_block
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M + N + K)
    x, r = torch.randn(M, K).bfloat16(), torch.randn(M, N).bfloat16()
    w, s = quantize_fp8_block(torch.randn(N, K) * 0.05, (64, 128))
    kw = dict(residual=r) if epi == "residual" else dict(epi=ref.EPI_SILU_MUL) if epi == "glu" else {}
    want = ref.linear_fp8(x, w, s, **kw)
    kw = {n: v.cuda() if isinstance(v, torch.Tensor) else v for n, v in kw.items()}
    got = [cu.linear_fp8(x.cuda(), w.cuda(), s.cuda(), **kw).cpu() for _ in range(2)]
    cu.check_status(torch.device("cuda", 0))
    assert float((got[0].float() - want.float()).norm() / want.float().norm()) < 2 ** -7
    assert torch.equal(*got)        # added in K order


def test_row_quantisation_into_words():
    """A result that starts on 4 bytes, not on 8."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(2)
    T, K = 5, 256
    x = torch.randn(T, K).bfloat16().cuda()
    want, scales = cu.quant_fp8_rows(x)
    buf, s = torch.zeros(T * K + 8, dtype=torch.uint8, device="cuda"), torch.empty_like(scales)
    assert cu._lib.lib().pxl_quant_fp8_rows(x.data_ptr(), K, buf.data_ptr() + 4, s.data_ptr(), T, K,
                                            torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(buf[4:-4], want.view(torch.uint8).flatten()) and torch.equal(s, scales)
    assert int(buf[:4].sum()) == 0 and int(buf[-4:].sum()) == 0


@pytest.mark.parametrize("M", [1, 7, 31, 32, 33, 64, 97, 127, 128])
@pytest.mark.parametrize("N,K,epi", [(39168, 256, "glu"), (128, 2048, "plain")])
def test_fp8_product_of_part_of_a_tile(M, N, K, epi):
    """Boxes of fewer than 128 rows and warps without a row, with a tile per CTA and split over a cluster; rows of A that follow the
    last one in memory are no numbers."""
    from parallax_b200.loader.quant import quantize_fp8_block
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M + N)
    x = torch.full((136, K), float("nan")).bfloat16().cuda()
    x[:M] = torch.randn(M, K).bfloat16().cuda()
    w, s = quantize_fp8_block(torch.randn(N, K, device="cuda") * 0.05, (64, 128))
    kw = dict(epi=ref.EPI_SILU_MUL) if epi == "glu" else {}
    want, got = ref.linear_fp8(x[:M], w, s, **kw), cu.linear_fp8(x[:M], w, s, **kw)
    cu.check_status(torch.device("cuda", 0))
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("M", [5, 8, 61, 120, 128])
def test_gated_bf16_product_of_part_of_a_tile(M):
    """The same for bf16 gate / up products, whose rows stay in the first operand's place."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M)
    x = torch.full((136, 512), float("nan")).bfloat16().cuda()
    x[:M] = torch.randn(M, 512).bfloat16().cuda()
    w = (torch.randn(38400, 512) * 0.05).bfloat16().cuda()
    y = x[:M].float() @ w.float().t()
    y = y.view(M, -1, 2, 64)
    want = (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(M, -1)
    got = cu.linear(x[:M], w, epi=ref.EPI_SILU_MUL)
    cu.check_status(torch.device("cuda", 0))
    assert float((got.float() - want).norm() / want.norm()) < 2 ** -8
