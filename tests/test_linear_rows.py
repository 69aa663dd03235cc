"""Streaming linears of one to eight rows on both sides of the widths where a warp's share of the matrix changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("N", [2367, 2368, 2369, 3552, 3553, 4736, 4737, 7104, 7105, 9473])
@pytest.mark.parametrize("gated", [False, True])
def test_rows_together_and_alone(N, gated):
    from ironpangu_b200.ops import decode as K

    g = torch.Generator().manual_seed(N)
    k, eps = 264, 1e-5
    w = (torch.randn(N * (1 + gated), k, generator=g) * 0.05).to(BF16).cuda()
    x, gain = torch.randn(8, k, generator=g).to(BF16).cuda(), (torch.rand(k, generator=g) + 0.5).to(BF16).cuda()
    xn = x.float()
    xn = (xn * torch.rsqrt(xn.square().mean(-1, keepdim=True) + eps) * gain.float()).to(BF16).double()
    y = xn @ w.double().T
    if gated:
        a, u = y[:, :N].float().to(BF16).double(), y[:, N:].float().to(BF16).double()
        y = a * torch.sigmoid(a) * u
    alone = torch.cat([K.gemv(x[t:t + 1], w, norm_w=gain, eps=eps, swiglu=gated) for t in range(8)])
    for T in (2, 3, 4, 5, 8):
        assert torch.equal(K.gemv(x[:T], w, norm_w=gain, eps=eps, swiglu=gated), alone[:T])
    # the result's rounding to bf16; an operand a rounding of bf16 apart (2^-8 of |x| <= 5 beside |w| <= 0.25: 0.005; gated: of one projection, times the other
    # of up to 4, and the projections' own roundings of 2^-8 each)
    tol = dict(rtol=2 ** -8, atol=0.005) if not gated else dict(rtol=3 * 2 ** -8, atol=0.02)
    torch.testing.assert_close(alone.double(), y, **tol)
