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
