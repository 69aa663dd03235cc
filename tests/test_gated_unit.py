"""The SiLU unit of gated projections over every bf16 gate, in each of the kernels that store it, against double precision."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _all_gates():
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(BF16)
    return g[torch.isfinite(g)].cuda()


@pytest.mark.parametrize("rows,F", [(255, 8), (65536, 8), (65536, 128)])        # few rows, one CTA a tile, CTA pairs
def test_every_gate(rows, F):
    from ironpangu_b200.ops import stream_norm as N

    g = _all_gates()
    a = torch.zeros(g.numel(), 8, dtype=BF16, device="cuda")
    a[:, 0], a[:, 1] = g, 1
    w = torch.zeros(2 * F, 8, dtype=BF16, device="cuda")
    w[:F, 0], w[F:, 1] = 1, 1
    out = torch.empty(g.numel(), F, dtype=BF16, device="cuda")
    for r in range(0, g.numel(), rows):
        N.gated_linear(a[r:r + rows], w, N.SILU, out[r:r + rows])
    z = g.double()
    want = z / (1 + torch.exp(-z))
    # one rounding to bf16 (half of 2^-7 of the value below), and before it an exponential whose error grows with its argument: 2^-17 at 88
    ulp = 2.0 ** (torch.frexp(want).exponent.double() - 8)
    off = (out.double() - want[:, None]).abs().amax(1)
    ok = off <= 0.5 * ulp + 2.0 ** -16 * want.abs()
    tiny = want.abs() < 2.0 ** -124                 # next to the smallest values of bf16
    assert bool((ok | tiny).all()), g[~(ok | tiny)][:8]
    assert bool((off[tiny] <= 2.0 ** -124).all())


def test_infinite_gate():
    from ironpangu_b200.ops import stream_norm as N

    a = torch.zeros(4, 8, dtype=BF16, device="cuda")
    a[:, 0], a[:, 1] = 3e38, 1
    w = torch.zeros(16, 8, dtype=BF16, device="cuda")
    w[:8, 0], w[8:, 1] = 4, 2                       # the projection overflows
    out = torch.empty(4, 8, dtype=BF16, device="cuda")
    N.gated_linear(a, w, N.SILU, out)
    assert bool((out == float("inf")).all())
