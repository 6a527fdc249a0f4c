"""Products of 129 to 1024 rows with a residual, a bias or fp32 results: their plan counts what the last tile does with them."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_plan_with_a_residual():
    from parallax_b200.ops import cuda as cu

    for M, N in ((256, 512), (512, 128), (1000, 128), (129, 512)):
        assert cu.gemm_mid_m_plan(M, N, 2048, cu.EPI_RESIDUAL)[1] > 1


@pytest.mark.parametrize("M,N,K", [(256, 512, 2048), (1000, 128, 2048), (129, 504, 2056), (700, 2048, 768), (384, 5120, 1024)])
@pytest.mark.parametrize("form", ["bias", "fp32", "residual and bias"])
def test_products(M, N, K, form):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M + N)
    x, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") / K ** 0.5).bfloat16()
    b, r = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
    want = x.double() @ w.double().t()
    if form == "fp32":
        got = cu.linear(x, w, epi=cu.EPI_F32)
    elif form == "bias":
        got, want = cu.linear(x, w, bias=b), want + b.double()
    else:
        got, want = cu.linear(x, w, bias=b, residual=r), want + b.double() + r.double()
    cu.check_status(torch.device("cuda", 0))
    # bf16 results: half a last place is at most 2^-8 of a value; fp32 sums of K products: far below 2^-17
    assert float((got.double() - want).norm() / want.norm()) < (2 ** -17 if form == "fp32" else 2 ** -8)
