"""RMS norm at the lines between its kernels: rows, columns, with and without a residual."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H", [(1, 8), (16, 1536), (511, 264), (512, 2056), (1535, 512), (1536, 512), (1536, 520), (2047, 72), (2048, 2048),
                                 (3, 8192), (3, 8200), (3, 16384), (3, 16392), (1023, 8200), (1024, 8200), (1024, 8192)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_norm(T, H, with_residual):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(T)
    x, w, r = torch.randn(T, H).bfloat16(), torch.randn(H).bfloat16(), torch.randn(T, H).bfloat16()
    stream = r.cuda() if with_residual else None
    got = cu.rmsnorm(x.cuda(), w.cuda(), 1e-6, residual=stream, w_offset=1.0).cpu().double()
    if with_residual:
        x = x + r                      # rounded to bf16: the new residual
        assert torch.equal(stream.cpu(), x)
    f = x.double()
    want = f * torch.rsqrt((f * f).mean(1, keepdim=True) + 1e-6) * (w.double() + 1.0)
    # rounded to bf16 (half of a last place: 2^-8 at most); the sum of squares, the root (2^-22) and three products in fp32, of which
    # the offset weight loses up to 2^-24 of its terms
    size = (f * torch.rsqrt((f * f).mean(1, keepdim=True))).abs() * (1.0 + w.double().abs())
    assert bool(((got - want).abs() <= 2 ** -8 * want.abs() + 2 ** -18 * size).all())
