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
