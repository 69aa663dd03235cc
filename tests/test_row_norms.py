"""Row kernels at the edges of their pieces: the gated group norm in pieces of four and element by element, the output norm at the width where a row's
CTA grows from 128 to 256 threads, against PyTorch in double precision."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("groups,n", [(3, 4), (9, 124), (8, 128), (2, 132), (1, 512), (1, 516), (2, 1024), (1, 2044), (1, 2048), (1, 2052), (5, 6)])
@pytest.mark.parametrize("off", [0, 2, 4])                     # elements between a 16-byte boundary and the rows of gate and result
def test_gated_group_norm(groups, n, off):
    from ironpangu_b200.ops import stream_norm as N

    T, W, eps = 5, groups * n, 1e-3
    g = torch.Generator().manual_seed(n + off)
    o, w = torch.randn(T, W, generator=g), torch.rand(W, generator=g) + 0.5
    gate = (torch.randn(T, W + 8, generator=g) * 3).to(BF16).cuda()[:, off:off + W]
    out = torch.zeros(T, W + 8, dtype=BF16, device="cuda")
    x = o.double().view(T, groups, n)
    unit = (x / (x.square().mean(-1, keepdim=True) + eps).sqrt()).reshape(T, W)
    for act, f in (("silu", torch.nn.functional.silu), ("sigmoid", torch.sigmoid)):
        for gain in (None, w):
            N.group_norm_gate(o.cuda(), gate, act, eps, out[:, off:off + W], groups, None if gain is None else gain.cuda())
            want = unit * f(gate.cpu().double()) * (1.0 if gain is None else gain.double())
            # one rounding to bf16 (2^-8); fast exponential and quotient, f32 sums: 1e-5 of the value
            torch.testing.assert_close(out[:, off:off + W].cpu().double(), want, rtol=2 ** -8 + 1e-5, atol=1e-6)
    assert int(out[:, :off].count_nonzero()) == 0 and int(out[:, off + W:].count_nonzero()) == 0


@pytest.mark.parametrize("D", [4, 508, 512, 516, 2044, 2046, 2048, 2052, 4096, 4100])
def test_output_norm(D):
    from ironpangu_b200.ops import stream_norm as N

    T, eps = 3, 1e-3
    g = torch.Generator().manual_seed(D)
    y, x, w, w2 = torch.randn(T, D, generator=g), torch.randn(T, D, generator=g), torch.rand(D, generator=g) + 0.5, torch.rand(D, generator=g) + 0.5
    rms = lambda v: v / (v.square().mean(-1, keepdim=True) + eps).sqrt()
    want = x.double() + rms(y.double()) * w.double()
    xd, xa = x.cuda(), torch.zeros(T, D, device="cuda")
    N.post_norm_add(y.cuda(), w.cuda(), eps, xd, xa, w2.cuda())
    # f32: a sum of D squares in pieces (a few 2^-24 of it), four roundings of terms up to 6
    torch.testing.assert_close(xd.cpu().double(), want, rtol=2e-6, atol=2e-6)
    torch.testing.assert_close(xa.cpu().double(), rms(want) * w2.double(), rtol=4e-6, atol=4e-6)
