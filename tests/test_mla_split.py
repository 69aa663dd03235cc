"""Split-KV latent attention on the tensor cores at the edges of its tiles (32 keys, 16 and 32 heads) against PyTorch in double precision."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
LATENT, ROPE = 512, 64


@pytest.mark.parametrize("heads", [4, 8, 16, 20, 32, 64])
@pytest.mark.parametrize("contexts,splits,sinks,window", [([1], 1, 0, 0), ([31, 32, 33], 3, 0, 0), ([64, 65, 500, 2], 4, 3, 0), ([400, 90], 8, 0, 70), ([300] * 9, 64, 2, 128)])
def test_heads_and_lengths(heads, contexts, splits, sinks, window):
    from ironpangu_b200.ops import prefill as P
    from ironpangu_b200.ops import _lib
    import ctypes as C

    g = torch.Generator(device="cuda").manual_seed(heads + len(contexts) + sinks)
    T, page = len(contexts), 16
    most = (max(contexts) + page - 1) // page
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    cache, q, sink = rand(T * most, page, LATENT + ROPE), rand(T, heads, LATENT + ROPE), rand(max(1, sinks), LATENT + ROPE)
    table = torch.randperm(T * most, generator=g, device="cuda").int().view(T, most)
    pos = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    slots = torch.arange(T, dtype=torch.int32, device="cuda")
    scratch = torch.empty(T * heads * splits * (LATENT + 2), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    scale, kps = (LATENT + ROPE) ** -0.5, 24
    rc = _lib.load().ifab_mla_decode_attention(q.data_ptr(), cache.data_ptr(), pos.data_ptr(), slots.data_ptr(), table.data_ptr(), most, page, T * most,
                                               sink.data_ptr() if sinks else None, sinks, window, scale, T, heads, LATENT, ROPE, kps, splits, scratch.data_ptr(),
                                               scratch.numel() * 4, None, 128, 128, None, 0, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    parts = scratch.view(T, heads, splits, LATENT + 2).double()
    for t, c in enumerate(contexts):
        n = min(c, window) if window else c
        rows = torch.cat([sink[:sinks], cache[table[t].long()].reshape(-1, LATENT + ROPE)[c - n:c]]).double()
        s = q[t].double() @ rows.T * scale
        ref = torch.softmax(s, -1) @ rows[:, :LATENT]
        used = min(splits, (len(rows) + kps - 1) // kps)
        m, l, acc = parts[t, :, :used, LATENT], parts[t, :, :used, LATENT + 1], parts[t, :, :used, :LATENT]
        w = torch.exp(m - m.max(-1, keepdim=True).values)
        out = (w[..., None] * acc).sum(1) / (w * l).sum(-1)[:, None]
        # scores, weights and sums in f32: 2^-18 of values up to 5
        torch.testing.assert_close(out, ref, rtol=0, atol=2e-5)
    assert int(status) == 0


@pytest.mark.parametrize("heads,n,splits", [(8, 60, 1), (8, 500, 1), (16, 1000, 1), (32, 1000, 16), (32, 4000, 8)])
def test_parts_are_f32_sums(heads, n, splits):
    """Maxima, sums and outputs as the kernel leaves them, before any rounding to bf16, against double precision."""
    from ironpangu_b200.ops import _lib

    g = torch.Generator(device="cuda").manual_seed(heads + n)
    pages = (n + 15) // 16
    cache, q = (torch.randn(*s, generator=g, device="cuda").to(BF16) for s in ((pages, 16, LATENT + ROPE), (1, heads, LATENT + ROPE)))
    table, pos, slot = torch.arange(pages, dtype=torch.int32, device="cuda"), torch.tensor([n - 1], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.empty(heads * splits * (LATENT + 2), device="cuda")
    assert _lib.load().ifab_mla_decode_attention(q.data_ptr(), cache.data_ptr(), pos.data_ptr(), slot.data_ptr(), table.data_ptr(), pages, 16, pages, None, 0, 0,
                                                 (LATENT + ROPE) ** -0.5, 1, heads, LATENT, ROPE, (n + splits - 1) // splits, splits, scratch.data_ptr(), scratch.numel() * 4, None,
                                                 128, 128, None, 0, None, torch.cuda.current_stream().cuda_stream) == 0
    parts = scratch.view(heads, splits, LATENT + 2).double()
    w = torch.exp(parts[..., LATENT] - parts[..., LATENT].max(-1, keepdim=True).values)
    out = (w[..., None] * parts[..., :LATENT]).sum(1) / (w * parts[..., LATENT + 1]).sum(-1)[:, None]
    rows = cache.view(-1, LATENT + ROPE)[:n].double()
    ref = torch.softmax(q[0].double() @ rows.T * (LATENT + ROPE) ** -0.5, -1) @ rows[:, :LATENT]
    # scores of up to 5 with a few roundings to 2^-24 of them, weights 2^-22 off at most, sums of up to 4000 terms: 2e-7 as f32 sums in any order are; where the tensor
    # cores add up along a whole row, cutting off, 1.5e-6 and more
    assert float((out - ref).norm() / ref.norm()) < 4e-7


@pytest.mark.parametrize("nope", [32, 64, 128])
def test_absorbed_query_is_the_one_of_a_row_alone(nope):
    """The order of its sums, bit for bit: 32 parts of nope / 32 elements in sequence, then a tree of halves. The one-launch kernel of one and two rows has it."""
    from ironpangu_b200.ops import decode as K

    T, H, vdim = 3, 5, 32
    g = torch.Generator(device="cuda").manual_seed(nope)
    q = torch.randn(T, H * (nope + ROPE), generator=g, device="cuda").to(BF16)
    w = torch.randn(H, nope + vdim, LATENT, generator=g, device="cuda").to(BF16)
    out = K.mla_q_absorb(q, w, torch.zeros(T, dtype=torch.int32, device="cuda"), nope=nope, rope=ROPE, theta=1e4)
    part = torch.zeros(T, H, 32, LATENT, device="cuda")
    for j in range(nope // 32):                    # a product of two bf16 values is exact in f32, so this is what a fused multiply-add rounds to
        d = torch.arange(32, device="cuda") * (nope // 32) + j
        prod = q.view(T, H, -1)[:, :, d].double()[..., None] * w[:, d].double()[None]
        part = (part.double() + prod).float()
    while part.shape[2] > 1:
        part = part[:, :, :part.shape[2] // 2] + part[:, :, part.shape[2] // 2:]
    assert torch.equal(out.view(T, H, -1)[..., :LATENT], part[:, :, 0].to(BF16))
