"""Products on both sides of the lines between their kernels (shared K over a cluster, one CTA a tile, CTA pairs with tiles of 128, 192 and 256 columns), with
remainders in rows and columns, against PyTorch in double precision."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _rand(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda").to(BF16)


def _slack(a, b):
    """What f32 sums in any order may be off by, the tensor cores' sums being cut off and not rounded: 2^-20 of the sum of magnitudes."""
    return float((a.double().abs() @ b.double().abs().T).max()) * 2.0 ** -20 + 1e-6


# one CTA a tile from 33 rows of more than 148 tiles of 128 columns on (20000), and where the rows are many beside K in a quarter of that (5000: tiles of 32
# columns, 12288: of 64); clusters of 8 with two K blocks each from 65 rows on (1024 x 1024); 129 rows and more to the pairs or to clusters by what is loaded
@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("M,N,K", [(32, 20000, 128), (33, 20000, 128), (128, 20008, 72), (129, 20000, 128), (12, 5000, 256), (13, 5000, 256), (128, 5000, 264), (100, 12288, 128),
                                   (64, 1024, 1024), (65, 1024, 1024), (128, 1032, 1096), (129, 1024, 1024), (255, 8192, 512), (255, 8200, 512), (200, 264, 2048), (130, 250, 128),
                                   (384, 3072, 2048), (256, 2112, 4096), (700, 2048, 4096), (1030, 512, 2048)])
def test_either_side_of_a_line(M, N, K, fixed):
    from ironpangu_b200.ops import gemm as G

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = _rand(g, M, K + 8)[:, :K], _rand(g, N, K)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = a.double() @ b.double().T
    out = torch.full((M + 1, N + 4), 7.0, device="cuda")
    G.gemm(a, b, out=out[:M, :N], status_ptr=status.data_ptr(), fixed=fixed)
    torch.testing.assert_close(out[:M, :N].double(), ref, rtol=0, atol=_slack(a, b))
    assert bool((out[M:] == 7).all()) and bool((out[:, N:] == 7).all())
    res = _rand(g, M, N)
    y = G.gemm(a, b, residual=res, status_ptr=status.data_ptr(), fixed=fixed)
    want = ref + res.double()
    # the product counts as a bf16 row, so does the sum: a rounding to bf16 is off by at most 2^-8 of the value
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * (ref.abs() + want.abs()) + _slack(a, b)).all())
    assert int(status) == 0


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("M,F,K", [(96, 12000, 64), (97, 12000, 64), (100, 2440, 128), (16, 2440, 512), (128, 2432, 512), (129, 512, 1024), (255, 6144, 256), (255, 6152, 256), (256, 512, 2048),
                                   (300, 520, 2048), (700, 1024, 4096), (1024, 72, 1024)])
def test_gated_either_side_of_a_line(M, F, K, fixed):
    from ironpangu_b200.ops import stream_norm as N

    g = torch.Generator(device="cuda").manual_seed(M + F + K)
    a, w = _rand(g, M, K), _rand(g, 2 * F, K) * K ** -0.5
    out = torch.full((M + 1, F + 8), 7.0, dtype=BF16, device="cuda")
    N.gated_linear(a, w, N.SILU, out[:M, :F], fixed=fixed)
    gate, up = (a.double() @ t.double().T for t in (w[:F], w[F:]))
    want = torch.nn.functional.silu(gate) * up
    # both projections and the result are rounded to bf16 (2^-8 of a value at most); silu is at most 1.1 times as steep as its argument; 2 % for
    # products of the three and the f32 sums
    bound = 1.02 * 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 2 * want.abs()) + 1e-4
    assert bool(((out[:M, :F].double() - want).abs() <= bound).all())
    assert bool((out[M:] == 7).all()) and bool((out[:, F:] == 7).all())


# with 74 pairs: 1000 x 3104 and 1505 x 2048 take tiles of 192 columns (the last one of 32 and of 128), 1000 x 768 of 128, 2000 x 12224 and 1000 x 4128 of 256
@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("M,N,K", [(1000, 3104, 200), (1505, 2048, 136), (1000, 768, 72), (2000, 12224, 64), (1000, 4128, 64)])
def test_pairs_of_every_width(M, N, K, persistent):
    from ironpangu_b200.ops.gemm import gemm_2sm

    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = _rand(g, M, K), _rand(g, N, K)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = gemm_2sm(a, b, out_f32=True, status_ptr=status.data_ptr(), persistent=persistent)
    torch.testing.assert_close(out.double(), a.double() @ b.double().T, rtol=0, atol=_slack(a, b))
    assert int(status) == 0


@pytest.mark.parametrize("M,F,K", [(2000, 6112, 64), (1000, 1568, 200), (300, 160, 136), (512, 6144, 128)])        # tiles of 256, 192, 128 and 192 columns
def test_gated_pairs_of_every_width(M, F, K):
    from ironpangu_b200.ops.gemm import gemm_swiglu

    g = torch.Generator(device="cuda").manual_seed(M + F)
    a, w = _rand(g, M, K), _rand(g, 2 * F, K) * K ** -0.5
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = gemm_swiglu(a, w, status_ptr=status.data_ptr())
    gate, up = (a.double() @ t.double().T for t in (w[:F], w[F:]))
    want = torch.nn.functional.silu(gate) * up
    bound = 1.02 * 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 2 * want.abs()) + 1e-4
    assert bool(((out.double() - want).abs() <= bound).all()) and int(status) == 0
