"""Expert kernels of a step of several tokens: tokens that share experts, and a CTA per token at one rank, give exactly what every token gives alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("T,E,topk,D,F,Fs", [(2, 4, 2, 256, 64, 64), (8, 4, 3, 512, 144, 80), (5, 16, 8, 1024, 256, 0), (8, 96, 8, 4096, 1536, 1536), (11, 6, 2, 256, 48, 48)])
def test_tokens_together_equal_tokens_alone(fp8, T, E, topk, D, F, Fs):
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.parallel.fabric import Fabric

    g = torch.Generator(device="cuda").manual_seed(T + E + D)
    rand = lambda *s: (torch.randn(*s, generator=g, device="cuda") * 0.05).to(BF16)
    x, gu, dn = rand(T, D) * 20, rand(E, 2 * F, D), rand(E, D, F)
    sgu, sdn = (rand(2 * Fs, D), rand(D, Fs)) if Fs else (None, None)
    ids = torch.stack([torch.randperm(E, generator=g, device="cuda")[:topk] for _ in range(T)]).int()
    wts = torch.rand(T, topk, generator=g, device="cuda")
    res = rand(T, D) * 10
    fab = Fabric(0, 1)
    q = (lambda w: None if w is None else K.quantize_fp8_block(w)) if fp8 else (lambda w: w)
    gu, dn, sgu, sdn = q(gu), q(dn), q(sgu), q(sdn)

    def gate_up(a, b):
        fn = K.moe_gate_up_fp8 if fp8 else K.moe_gate_up
        return fn(x[a:b], ids[a:b], gu, 0, w_shared_gu=sgu, act=torch.zeros(b - a, topk + 1, F, dtype=BF16, device="cuda"))

    def down(act, a, b):
        fn = K.moe_down_allreduce_fp8 if fp8 else K.moe_down_allreduce
        return fn(act[a:b].contiguous(), ids[a:b], wts[a:b], dn, 0, fab, w_shared_down=sdn, residual=res[a:b], out=torch.empty(b - a, D, dtype=BF16, device="cuda"))

    act = gate_up(0, T)
    assert torch.equal(act, torch.cat([gate_up(t, t + 1) for t in range(T)]))
    if T <= 8:
        assert torch.equal(down(act, 0, T), torch.cat([down(act, t, t + 1) for t in range(T)]))
    assert fab.status() == 0
    fab.close()


@pytest.mark.parametrize("fp8", [True, False])
@pytest.mark.parametrize("T", [1, 2, 8])
def test_rows_too_wide_are_refused_for_any_number_of_tokens(fp8, T):
    """Rows of the down projection: 296 CTAs of 32 columns at the most, at one rank too."""
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.parallel.fabric import Fabric

    fab = Fabric(0, 1)
    E, topk, F = 2, 1, 32
    fn = K.moe_down_allreduce_fp8 if fp8 else K.moe_down_allreduce
    for D in (296 * 32, 296 * 32 + 8):
        dn = torch.zeros(E, D, F, dtype=BF16, device="cuda")
        args = (torch.zeros(T, topk + 1, F, dtype=BF16, device="cuda"), torch.zeros(T, topk, dtype=torch.int32, device="cuda"), torch.ones(T, topk, device="cuda"),
                K.quantize_fp8_block(dn) if fp8 else dn, 0, fab)
        out = torch.ones(T, D, dtype=BF16, device="cuda")
        if D > 296 * 32:
            with pytest.raises(RuntimeError):
                fn(*args, out=out)
        else:
            fn(*args, out=out)
            assert int(out.count_nonzero()) == 0
    fab.close()
