"""Linears of one to eight rows as a stream through rings, at the edges of their shares: more SMs than rows of the matrix, remainders of eight rows, of a warp's columns and of
a ring; rows of x that fit shared memory and that do not."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("gated,norm", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("N,K,T", [(1, 8, 2), (7, 520, 1), (147, 1024, 8), (149, 1032, 3), (2368, 1544, 5), (2999, 2048, 8), (5000, 264, 2), (300, 6144, 8), (300, 16384, 8), (64, 16392, 1), (9000, 512, 11)])
def test_shares_and_remainders(N, K, T, gated, norm):
    from ironpangu_b200.ops import decode as D

    g = torch.Generator(device="cuda").manual_seed(N + K + T)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w = rand(T, K + 8).to(BF16)[:, :K], (rand(N * (1 + gated), K) * K ** -0.5).to(BF16)
    gain = (rand(K) * 0.1 + 1).to(BF16) if norm else None
    operand = x.float()
    if norm:
        operand = (operand * torch.rsqrt(operand.square().mean(-1, keepdim=True) + 1e-6) * gain.float()).to(BF16).float()
    ref = operand.double() @ w.double().T
    # f32 sums; a norm in f32 may round an operand to the next bf16 value (2^-8 of it) in another order of its sum: a few of K
    slack = float((operand.double().abs() @ w.double().abs().T).max()) * (2.0 ** -20 + (2.0 ** -8 * K ** -0.5 if norm else 0.0)) + 1e-6
    if gated:
        out = torch.full((T + 1, N + 3), 7.0, dtype=BF16, device="cuda")
        D.gemv(x, w, norm_w=gain, eps=1e-6, swiglu=True, out=out[:T, :N], rings=True)
        gate, up = ref[:, :N], ref[:, N:]
        want = torch.nn.functional.silu(gate) * up
        bound = 1.02 * 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 2 * want.abs()) + slack * (2 * up.abs() + 2 * gate.abs() + 1)
        assert bool(((out[:T, :N].double() - want).abs() <= bound).all())
    else:
        out = torch.full((T + 1, N + 3), 7.0, device="cuda")
        D.gemv(x, w, norm_w=gain, eps=1e-6, out=out[:T, :N], rings=True)
        torch.testing.assert_close(out[:T, :N].double(), ref, rtol=0, atol=slack)
        res = rand(T, N).to(BF16)
        y = res.clone()
        D.gemv(x, w, norm_w=gain, eps=1e-6, residual=y, out=y, rings=True)          # in place
        want = ref + res.double()
        assert bool(((y.double() - want).abs() <= 2.0 ** -8 * (ref.abs() + want.abs()) + slack).all())
    assert bool((out[T:] == 7).all()) and bool((out[:, N:] == 7).all())
    alone = torch.cat([D.gemv(x[t:t + 1], w, norm_w=gain, eps=1e-6, swiglu=gated, rings=True) for t in range(T)])
    assert torch.equal(D.gemv(x, w, norm_w=gain, eps=1e-6, swiglu=gated, rings=True), alone)          # the bits that a row has alone


@pytest.mark.parametrize("T,V,K", [(1, 31, 64), (1, 33, 1032), (2, 5000, 512), (3, 700, 520), (8, 17, 64), (8, 9000, 4104)])
def test_greedy_head(T, V, K):
    from ironpangu_b200.ops import decode as D
    from ironpangu_b200.parallel.fabric import Fabric

    g = torch.Generator(device="cuda").manual_seed(T + V + K)
    x, w = torch.randn(T, K, generator=g, device="cuda").to(BF16), (torch.randn(V, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    w[V // 2] = w[0]                                     # equal logits: the lowest id
    fab = Fabric(0, 1)
    for keep in (True, False):
        logits = torch.full((T, V), 7.0, device="cuda") if keep else None
        ids = D.lm_head_argmax(x, w, fab, logits=logits)
        ref = x.double() @ w.double().T
        slack = float((x.double().abs() @ w.double().abs().T).max()) * 2.0 ** -20 + 1e-6
        best = ref.max(-1).values
        assert bool((best - ref.gather(1, ids.long()[:, None])[:, 0] <= 2 * slack).all())
        assert not bool((ids == V // 2).any()) or V // 2 == 0
        if keep:
            torch.testing.assert_close(logits.double(), ref, rtol=0, atol=slack)
    assert fab.status() == 0
    fab.close()


# operands made of a norm's output and a residual, of normalised groups with gates, and plain rows too long for shared memory
@pytest.mark.parametrize("T", [1, 2, 3])
@pytest.mark.parametrize("K,N,groups", [(192, 328, 6), (2048, 150, 16), (4096, 1000, 1), (4104, 147, 3), (9000, 77, 9)])
def test_operands_of_norms_and_gates(T, K, N, groups):
    from ironpangu_b200.ops import stream_norm as S

    g = torch.Generator(device="cuda").manual_seed(K + N + T)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    w, y, x, gain, eps = (rand(N, K) * K ** -0.5).to(BF16), rand(T, K), rand(T, K) * 4, rand(K) * 0.1 + 1, 1e-3
    rms = lambda v: v * torch.rsqrt(v.square().mean(-1, keepdim=True) + eps)

    def check(out, operand):
        # the operand may round to the next bf16 value (2^-8 of it) where its f32 norm ends a little off; f32 sums
        ref, scale = operand.to(BF16).double() @ w.double().T, float((operand.double().abs() @ w.double().abs().T).max())
        torch.testing.assert_close(out.double(), ref, rtol=0, atol=scale * (2.0 ** -20 + 2.0 ** -8 * K ** -0.5) + 1e-6)

    z, x_out = torch.empty(T, N, device="cuda"), torch.empty(T, K, device="cuda")
    S.gemv_post_norm(y, gain, eps, x, x_out, w, z, rings=True)
    want = x.double() + rms(y.double()) * gain.double()
    torch.testing.assert_close(x_out.double(), want, rtol=1e-5, atol=4e-6)
    check(z, want.float())
    gate = rand(T, K).to(BF16)
    S.gemv_group_norm(y, gate, "sigmoid", eps, w, z, groups, gain, rings=True)
    check(z, (rms(y.double().view(T, groups, -1)).view(T, K) * gain.double() * torch.sigmoid(gate.double())).float())
    xb = x.to(BF16)
    S.gemv_act(xb, w, z, rings=True)
    check(z, xb.float())
    bias, add = rand(N), rand(T, N)
    out = add.clone()
    S.gemv_act(xb, w, out, bias=bias, addend=out, rings=True)
    torch.testing.assert_close(out, z + bias + add, rtol=1e-5, atol=1e-5)


# heads of 128, 64, 40 and 2 columns; shares that end inside a head; rows that are not there, in the same sequence, and on a page outside the cache
@pytest.mark.parametrize("T,H,kv,hd,K", [(1, 16, 4, 128, 2048), (8, 8, 2, 64, 520), (3, 3, 3, 40, 256), (2, 5, 1, 2, 64)])
def test_projection_with_rotation_and_pages(T, H, kv, hd, K):
    from ironpangu_b200.ops import decode as D

    g = torch.Generator(device="cuda").manual_seed(T + hd + K)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, gain = rand(T, K).to(BF16), (rand((H + 2 * kv) * hd, K) * K ** -0.5).to(BF16), (rand(K) * 0.1 + 1).to(BF16)
    pages, table = 6, torch.tensor([[3, 1, 5], [0, 2, 77]], dtype=torch.int32, device="cuda")
    pos = torch.tensor([17, 18, 3, -1, 40, 0, 31, 5][:T], dtype=torch.int32, device="cuda")
    slots = torch.tensor([0, 0, 1, 1, 1, 1, 1, 0][:T], dtype=torch.int32, device="cuda")          # row 4 of eight: page 77
    def cache():
        return [torch.full((pages, 16, kv, hd), 7.0, dtype=BF16, device="cuda") for _ in range(2)]
    (k1, v1), (k2, v2) = cache(), cache()
    st1, st2 = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
    one = torch.full((T, (H + 2 * kv) * hd), 7.0, dtype=BF16, device="cuda")
    D.qkv_rows(x, w, gain, pos, slots, table, k1, v1, heads=H, kv_heads=kv, head_dim=hd, theta=1e4, eps=1e-6, out=one, status_ptr=st1.data_ptr())
    two = D.gemv(x, w, norm_w=gain, eps=1e-6, rings=True)
    if hd % 8 == 0:
        D.gqa_rope_kv_write(two, pos, slots, table, k2, v2, heads=H, kv_heads=kv, head_dim=hd, theta=1e4, status_ptr=st2.data_ptr())
        assert int(st1) == int(st2)
        # the same f32 products of bf16 values, added in f32 and rounded: at most one bf16 step where a sum ends beside a boundary
        for a, b in ((one[:, :H * hd], two[:, :H * hd]), (k1, k2), (v1, v2)):
            torch.testing.assert_close(a.float(), b.float(), rtol=2 ** -7, atol=2.0 ** -12)
        assert torch.equal(v1, v2)
    else:
        f = two.double().view(T, H + 2 * kv, hd)
        c, s = (t.float().to(BF16).double() for t in (torch.cos(pos.double()), torch.sin(pos.double())))
        for t in range(T):
            if int(pos[t]) >= 0:
                q = torch.stack([f[t, :H, 0] * c[t] - f[t, :H, 1] * s[t], f[t, :H, 1] * c[t] + f[t, :H, 0] * s[t]], -1).reshape(-1)
                torch.testing.assert_close(one[t, :H * hd].double(), q, rtol=2 ** -7, atol=2.0 ** -12)
    assert bool((one[:, H * hd:] == 7).all())


@pytest.mark.parametrize("T", [2, 8])
def test_columns_that_do_not_turn_are_copied(T):
    """Values, and queries of rows that are not there: an infinite or NaN column stays one column, as behind the projection and the rotation in launches of their own."""
    from ironpangu_b200.ops import decode as D

    H, kv, hd, K, page = 4, 2, 64, 256, 16
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, generator=g, device="cuda").to(BF16)
    w, gain = (torch.randn((H + 2 * kv) * hd, K, generator=g, device="cuda") * K ** -0.5).to(BF16), torch.ones(K, device="cuda", dtype=BF16)
    w[(H + kv) * hd + 3, 7] = float("inf")
    w[(H + kv) * hd + hd + hd // 2 + 5] = float("nan")
    w[9, 1] = float("inf")
    table = torch.arange(T, dtype=torch.int32, device="cuda")[:, None].contiguous()
    pos, slots = torch.arange(T, dtype=torch.int32, device="cuda") + 1, torch.arange(T, dtype=torch.int32, device="cuda")
    pos[1] = -1
    k1, v1, k2, v2 = (torch.full((T, page, kv, hd), 7.0, dtype=BF16, device="cuda") for _ in range(4))
    one = torch.empty(T, (H + 2 * kv) * hd, dtype=BF16, device="cuda")
    D.qkv_rows(x, w, gain, pos, slots, table, k1, v1, heads=H, kv_heads=kv, head_dim=hd, theta=1e4, eps=1e-6, out=one)
    two = D.gemv(x, w, norm_w=gain, eps=1e-6, rings=True)
    D.gqa_rope_kv_write(two, pos, slots, table, k2, v2, heads=H, kv_heads=kv, head_dim=hd, theta=1e4)
    torch.testing.assert_close(v1, v2, rtol=0, atol=0, equal_nan=True)
    torch.testing.assert_close(one[1, :H * hd], two[1, :H * hd], rtol=0, atol=0, equal_nan=True)
    assert int((~v1.isfinite()).sum()) == 2 * (T - 1) and int((~one[1, :H * hd].isfinite()).sum()) == 1
