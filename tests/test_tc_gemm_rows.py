"""Products of few rows (features as the rows of the MMA, K shared by a cluster) at the edges of their tiles against PyTorch in double precision."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _rand(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda").to(BF16)


def _slack(a, b):
    """What f32 sums in any order may be off by: 2^-22 of the sum of magnitudes."""
    return float((a.double().abs() @ b.double().abs().T).max()) * 2.0 ** -22 + 1e-6


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("M", [1, 7, 8, 16, 17, 33, 64, 65, 127, 128, 129, 200, 255, 300])
@pytest.mark.parametrize("N,K", [(8, 8), (100, 72), (128, 64), (129, 520), (1000, 1152), (2048, 6144), (3072, 2048)])
def test_any_rows_columns_and_depth(M, N, K, fixed):
    from ironpangu_b200.ops import gemm as G

    if M >= 256 and not (fixed and (N, K) == (2048, 6144)):
        pytest.skip("another kernel's")
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    a, b = _rand(g, M, K + 8)[:, :K], _rand(g, N, K)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = a.double() @ b.double().T
    out = torch.full((M + 1, N + 3), 7.0, device="cuda")                   # odd row stride, guard row and columns
    G.gemm(a, b, out=out[:M, :N], status_ptr=status.data_ptr(), fixed=fixed)
    torch.testing.assert_close(out[:M, :N].double(), ref, rtol=0, atol=_slack(a, b))
    assert bool((out[M:] == 7).all()) and bool((out[:, N:] == 7).all())
    res = _rand(g, M, N)
    y = G.gemm(a, b, residual=res, status_ptr=status.data_ptr(), fixed=fixed)
    # the product counts as a bf16 row, so does the sum: a rounding to bf16 is off by at most 2^-8 of the value
    want = ref + res.double()
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * (ref.abs() + want.abs()) + _slack(a, b)).all())
    assert int(status) == 0


@pytest.mark.parametrize("M", [1, 9, 64, 100, 190])
@pytest.mark.parametrize("F,K", [(8, 64), (72, 136), (192, 1024), (1000, 512)])
def test_gated_units_and_epilogues(M, F, K):
    from ironpangu_b200.ops import stream_norm as N

    g = torch.Generator(device="cuda").manual_seed(M + F + K)
    a, w = _rand(g, M, K), _rand(g, 2 * F, K) * K ** -0.5
    out = torch.empty(M, F, dtype=BF16, device="cuda")
    N.gated_linear(a, w, N.SILU, out, fixed=True)
    gate, up = (a.double() @ t.double().T for t in (w[:F], w[F:]))
    want = torch.nn.functional.silu(gate) * up
    # both projections and the result are rounded to bf16 (2^-8 of a value at most); silu is at most 1.1 times as steep as its argument; 2 % for
    # products of the three and the f32 sums
    bound = 1.02 * 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 2 * want.abs()) + 1e-5
    assert bool(((out.double() - want).abs() <= bound).all())
    bias = torch.randn(2 * F, generator=g, device="cuda")
    y = torch.empty(M, 2 * F, device="cuda")
    N.linear(a, w, y, "gelu_tanh", bias=bias, cap=2.0, fixed=True)
    z = torch.nn.functional.gelu(a.double() @ w.double().T + bias.double(), approximate="tanh")
    torch.testing.assert_close(y.double(), 2 * torch.tanh(z / 2), rtol=1e-4, atol=1e-4)
