"""Row kernels at the edges of their pieces: the gated group norm in pieces of four and element by element, the output norm at the widths and
numbers of rows where a row's CTA changes between 128 and 256 threads, against PyTorch in double precision."""
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
@pytest.mark.parametrize("T", [3, 591, 592, 700])              # 128 threads to a row from 592 rows on (four to an SM of 148), for up to 2048 columns
def test_output_norm(T, D):
    from ironpangu_b200.ops import stream_norm as N

    eps = 1e-3
    g = torch.Generator().manual_seed(D)
    y, x, w, w2 = torch.randn(T, D, generator=g), torch.randn(T, D, generator=g), torch.rand(D, generator=g) + 0.5, torch.rand(D, generator=g) + 0.5
    inv = lambda v: 1 / (v.square().mean(-1, keepdim=True) + eps).sqrt()
    want = x.double() + y.double() * inv(y.double()) * w.double()
    scale = inv(want) * w2.double()
    for second in (True, False):
        for dt in (torch.float32, BF16):
            xd, xa = x.cuda(), torch.zeros(T, D, dtype=dt, device="cuda")
            N.post_norm_add(y.cuda(), w.cuda(), eps, xd, xa, w2.cuda() if second else None)
            # f32: terms up to 8 with a relative error of 6 x 2^-24 (sum of squares in pieces, root, quotient, two products) and the rounding of a sum up to 13
            e = 6 * 2 ** -24 * 8 + 2 ** -24 * 13
            torch.testing.assert_close(xd.cpu().double(), want, rtol=0, atol=e)
            out, err = (want * scale, e * scale + 6 * 2 ** -24 * (want * scale).abs()) if second else (want, torch.full_like(want, e))
            if dt is BF16:
                err = err + 2 ** -8 * out.abs()
            assert bool(((xa.cpu().double() - out).abs() <= err).all())
