"""fp8 expert kernels that read an expert once for all of its tokens, where their lists and shares can go wrong: a token that names an expert twice, experts of other ranks, no
expert at all, columns and rows that are no multiple of a stage's, more rows than a CTA has at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _wide(w):
    q, s = w
    K = q.shape[-1]
    return q.view(torch.float8_e4m3fn).double() * s.double().repeat_interleave(128, -1)[..., :K]


@pytest.mark.parametrize("T,E,topk,D,F,Fs,shared", [(8, 3, 2, 64, 16, 16, True), (5, 300, 16, 2064, 144, 80, True), (3, 40, 4, 5008, 272, 0, False), (1, 8, 8, 9472, 128, 128, True), (8, 2, 1, 4112, 1040, 16, True)])
def test_lists_and_shares(T, E, topk, D, F, Fs, shared):
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.parallel.fabric import Fabric

    g = torch.Generator(device="cuda").manual_seed(T + E + D)
    rand = lambda *s: (torch.randn(*s, generator=g, device="cuda") * 0.05).to(BF16)
    x, res, gain = rand(T, D) * 20, rand(T, D) * 10, rand(D) + 1
    gu, dn = K.quantize_fp8_block(rand(E, 2 * F, D)), K.quantize_fp8_block(rand(E, D, F))
    sgu, sdn = (K.quantize_fp8_block(rand(2 * Fs, D)), K.quantize_fp8_block(rand(D, Fs))) if shared else (None, None)
    ids = torch.randint(-2, E + 2, (T, topk), generator=g, device="cuda").int()          # experts of nobody's among them
    if topk > 1:
        ids[0, 1] = ids[0, 0] = 1                                                          # one expert twice
    if T > 2:
        ids[2] = -1                                                                        # none at all
    wts = torch.rand(T, topk, generator=g, device="cuda")
    fab = Fabric(0, 1)
    calls = fab.calls()
    act = K.moe_gate_up_fp8(x, ids, gu, 0, norm_w=gain, w_shared_gu=sgu, act=torch.zeros(T, topk + 1, F, dtype=BF16, device="cuda"))
    y = K.moe_down_allreduce_fp8(act, ids, wts, dn, 0, fab, w_shared_down=sdn, residual=res)
    assert fab.calls() == calls + 1
    h = x.float()
    h = (h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-5) * gain.float()).to(BF16).double()
    GU, DN = _wide(gu), _wide(dn)
    for t in range(T):
        want, scale = torch.zeros(D, dtype=torch.float64, device="cuda"), torch.zeros(D, dtype=torch.float64, device="cuda")
        routes = [(k, GU[int(ids[t, k])], DN[int(ids[t, k])], float(wts[t, k]), F) for k in range(topk) if 0 <= int(ids[t, k]) < E]
        routes += [(topk, _wide(sgu), _wide(sdn), 1.0, Fs)] if shared else []
        used = {r[0] for r in routes}
        for k, wg, wd, c, f in routes:
            gate, up = wg[:f] @ h[t], wg[f:] @ h[t]
            a = torch.nn.functional.silu(gate) * up
            # both projections and their product are rounded to bf16 (2^-8 of a value at most, silu at most 1.1 times as steep); operands that a norm in f32 rounds to
            # the next bf16 value and f32 sums: 2^-8 K^-1/2 of the magnitudes
            slack = 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 2 * a.abs()) * 1.05 + (2 * up.abs() + 2 * gate.abs() + 1) * float((wg.abs() @ h[t].abs()).max()) * 2.0 ** -8 * D ** -0.5
            assert bool(((act[t, k, :f].double() - a).abs() <= slack).all())
            rows = act[t, k, :f].double()
            want += c * (wd @ rows)
            scale += c * (wd.abs() @ rows.abs())
        assert all(bool((act[t, k] == 0).all()) for k in range(topk + 1) if k not in used)
        total = want + res[t].double()
        assert bool(((y[t].double() - total).abs() <= 2.0 ** -8 * (want.abs() + total.abs()) + 2.0 ** -18 * scale + 1e-6).all())
    assert fab.status() == 0
    fab.close()


def test_threads_with_steps_of_different_widths():
    """The shared memory of a launch depends on the tokens; what the kernel is opened for does not, or one thread's launch would be refused for another's step."""
    import threading
    from ironpangu_b200.ops import decode as K

    from ironpangu_b200.ops import _lib

    E, topk, D, F = 4, 2, 4096, 16
    q, scales = K.quantize_fp8_block((torch.randn(E, 2 * F, D, device="cuda") * 0.05).to(BF16))
    fn, codes = _lib.load().ifab_moe_gate_up_decode_fp8, set()

    def steps(T):
        torch.cuda.set_device(0)
        with torch.cuda.stream(torch.cuda.Stream()):
            x, ids = torch.ones(T, D, dtype=BF16, device="cuda"), torch.zeros(T, topk, dtype=torch.int32, device="cuda")
            act = torch.zeros(T, topk + 1, F, dtype=BF16, device="cuda")
            args = (x.data_ptr(), D, None, 1e-5, ids.data_ptr(), T, D, F, topk, 0, E, q.data_ptr(), scales.data_ptr(), None, None, 0, act.data_ptr(),
                    torch.cuda.current_stream().cuda_stream)
            for _ in range(30):
                for _ in range(200):
                    codes.add(fn(*args))
                torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=steps, args=(T,)) for T in (1, 8) * 3]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert codes == {0}


def test_rows_too_wide_for_one_launch():
    """A launch has room for five rows of 9472 columns beside its rings: eight tokens take two, and each has what it has alone."""
    from ironpangu_b200.ops import decode as K

    test_lists_and_shares(8, 3, 2, 9472, 128, 128, True)
    g = torch.Generator(device="cuda").manual_seed(9472)
    rand = lambda *s: (torch.randn(*s, generator=g, device="cuda") * 0.05).to(BF16)
    T, E, topk, D, F = 8, 3, 2, 9472, 128
    x, gu, sgu, gain = rand(T, D) * 20, K.quantize_fp8_block(rand(E, 2 * F, D)), K.quantize_fp8_block(rand(2 * F, D)), rand(D) + 1
    ids = torch.randint(0, E, (T, topk), generator=g, device="cuda").int()
    act = K.moe_gate_up_fp8(x, ids, gu, 0, norm_w=gain, w_shared_gu=sgu)
    for t in range(T):
        assert torch.equal(act[t:t + 1], K.moe_gate_up_fp8(x[t:t + 1].clone(), ids[t:t + 1].clone(), gu, 0, norm_w=gain, w_shared_gu=sgu))


@pytest.mark.parametrize("E,rings", [(1024, True), (1030, True), (1030, None), (1024, False)])
def test_as_many_experts_as_a_list_has_and_more(E, rings):
    """1024 experts are what a list of routes has room for; more take the form that goes token by token, as small ones do. Small whole numbers, so that every sum is exact
    in either."""
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.parallel.fabric import Fabric

    g = torch.Generator(device="cuda").manual_seed(3)
    whole = lambda *s, top: torch.randint(-top, top + 1, s, generator=g, device="cuda").float()
    T, topk, D, F = 3, 4, 64, 16
    x, act_in = whole(T, D, top=1).to(BF16), whole(T, topk + 1, F, top=1).to(BF16)
    ids = torch.stack([torch.randperm(1020, generator=g, device="cuda")[:topk] for _ in range(T)]).int()
    ids[0] = torch.tensor([E - 1, E - 2, 0, 1023], device="cuda")
    wts = 2.0 ** -torch.randint(0, 3, (T, topk), generator=g, device="cuda").float()
    gu, dn = whole(E, 2 * F, D, top=4), whole(E, D, F, top=4)
    fp8 = lambda w: (w.to(torch.float8_e4m3fn).view(torch.uint8), torch.full((*w.shape[:-1], 1), 0.25, device="cuda"))
    fab = Fabric(0, 1)
    act = K.moe_gate_up_fp8(x, ids, fp8(gu), 0, rings=rings)
    y = K.moe_down_allreduce_fp8(act_in, ids, wts, fp8(dn), 0, fab)
    for t in range(T):
        total = torch.zeros(D, dtype=torch.float64, device="cuda")
        for k in range(topk):
            e = int(ids[t, k])
            got = (gu[e].double() @ x[t].double() * 0.25).to(BF16).double()
            a = torch.nn.functional.silu(got[:F]) * got[F:]
            assert bool(((act[t, k].double() - a).abs() <= a.abs() * (2.0 ** -8 + 2.0 ** -18)).all())          # one rounding, and silu in f32
            total += float(wts[t, k]) * (dn[e].double() @ act_in[t, k].double() * 0.25)
        assert torch.equal(y[t].double(), total.to(BF16).double())
    assert fab.status() == 0
    fab.close()
