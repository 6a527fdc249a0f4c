"""Large products whose nearly empty last wave of tiles goes in a launch of its own: the offsets of rows, residual and results into
it, and the kernels that tails of every size take, against the product in one launch."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (5889, 4096, 4096), (5892, 4096, 4096),         # one and four rows behind 46 tiles
    (5903, 4096, 4096), (6016, 4096, 4096),         # 15 and 128
    (4745, 1000, 4096),                             # columns that no tile divides
    (19244, 256, 4096),                             # 300: K split over a cluster
])
def test_tail_in_a_launch_of_its_own(M, N, K):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(M)
    x = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K]
    w = (torch.randn(N, K + 16, device="cuda") * 0.05).bfloat16()[:, :K]
    b, r = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N + 8, device="cuda").bfloat16()[:, :N]
    for kw, epi in ((dict(), 0), (dict(bias=b), 0), (dict(bias=b, residual=r), 0), (dict(bias=b), ref.EPI_F32)):
        dt = torch.float32 if epi else torch.bfloat16
        out, one = (torch.full((M + 1, N + 8), 7.0, dtype=dt, device="cuda") for _ in range(2))
        before = cu.launch_count
        cu.linear(x, w, epi=epi, out=out[:M, :N], **kw)
        assert cu.launch_count - before == 2
        cu.linear(x, w, epi=epi, out=one[:M, :N], bn=128, **kw)
        cu.check_status(torch.device("cuda", 0))
        assert bool((out[M] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
        # the same fp32 products in another order, rounded to bf16 (2^-9) where the result is: row by row, so that the tail's count
        err = (out[:M, :N].float() - one[:M, :N].float()).norm(dim=1) / one[:M, :N].float().norm(dim=1)
        assert float(err.max()) < (1e-5 if epi else 2 ** -8)


@pytest.mark.parametrize("M,N,K", [(1551, 5120, 8192), (2252, 5120, 8192), (5409, 1024, 3072)])
def test_tails_that_are_cheaper_in_the_last_wave(M, N, K):
    """Tails of hundreds of rows whose product is longer on its own than the wave that they share."""
    from parallax_b200.ops import _lib

    assert _lib.lib().pxl_gemm_bf16_launches(M, N, K, 0) == 1
