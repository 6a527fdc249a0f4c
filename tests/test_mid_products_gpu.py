"""Products of 129 to 1024 rows: the tile widths and clusters that the cost model picks."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(129, 2112, 7168), (256, 2112, 7168), (640, 1024, 3072), (144, 4096, 4096), (1000, 1024, 3072), (1024, 2112, 1032),
                                   (900, 6144, 1024), (130, 8, 4096)])
@pytest.mark.parametrize("epi", ["plain", "residual", "gated"])
def test_products(M, N, K, epi):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M + N)
    if epi == "gated" and N % 128:
        N += 128 - N % 128
    x, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") / K ** 0.5).bfloat16()
    want = x.double() @ w.double().t()
    if epi == "residual":
        r = torch.randn(M, N, device="cuda").bfloat16()
        got, want = cu.linear(x, w, residual=r), want + r.double()
    elif epi == "gated":
        got, p = cu.linear(x, w, epi=cu.EPI_SILU_MUL), want.view(M, -1, 2, 64)
        want = (torch.nn.functional.silu(p[:, :, 0]) * p[:, :, 1]).reshape(M, -1)
    else:
        got = cu.linear(x, w)
    cu.check_status(torch.device("cuda", 0))
    # the output is rounded to bf16: half a unit is at most 2^-8 of a value; sums in fp32 are far below
    assert float((got.double() - want).norm() / want.norm()) < 2 ** -8
