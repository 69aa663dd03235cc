"""Split-KV decode attention at the edges of its tiles (16 keys a warp, 64 a round) against PyTorch in double precision."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _reference(q, k, v, scale):
    """q [H, d], k / v [n, G, d]."""
    r = q.shape[0] // k.shape[1]
    s = torch.einsum("hd,nhd->hn", q.double(), k.double().repeat_interleave(r, 1)) * scale
    return torch.einsum("hn,nhd->hd", torch.softmax(s, -1), v.double().repeat_interleave(r, 1))


@pytest.mark.parametrize("hd,kv,group", [(64, 2, 1), (64, 2, 8), (128, 4, 4), (128, 1, 2), (128, 2, 8), (128, 3, 1), (256, 2, 4)])
@pytest.mark.parametrize("contexts,splits", [([1], 1), ([15, 16, 17], 4), ([63, 64, 65, 1], 64), ([1000, 129, 700, 2], 5), ([300] * 70, 64)])
def test_rows_of_any_length(hd, kv, group, contexts, splits):
    from ironpangu_b200.ops import decode as K

    g = torch.Generator(device="cuda").manual_seed(hd + kv + group + len(contexts))
    T, H, page = len(contexts), kv * group, 16
    most = (max(contexts) + page - 1) // page
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    kc, vc = rand(T * most, page, kv, hd), rand(T * most, page, kv, hd)
    q = rand(T, (H + 2 * kv) * hd)                                       # the query columns of a wider projection
    table = torch.randperm(T * most, generator=g, device="cuda").int().view(T, most)
    pos = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    slots = torch.arange(T - 1, -1, -1, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = K.gqa_decode_attention(q, kc, vc, pos, slots, table, heads=H, kv_heads=kv, head_dim=hd, scale=hd ** -0.5, keys_per_split=16, max_splits=splits,
                                 status_ptr=status.data_ptr())
    for t, c in enumerate(contexts):
        rows = table[int(slots[t])].long()
        k, v = kc[rows].reshape(-1, kv, hd)[:c], vc[rows].reshape(-1, kv, hd)[:c]
        ref = _reference(q[t, :H * hd].view(H, hd), k, v, hd ** -0.5).reshape(-1)
        # a rounding to bf16 (at most 2^-8 of the value), and weights of two bf16 terms (2^-16 of values up to 5)
        torch.testing.assert_close(out[t].double(), ref, rtol=2 ** -8, atol=1e-4)
    assert int(status) == 0


def test_caches_off_a_16_byte_boundary_and_pages_that_are_not_there():
    """Caches that start 8 bytes into their storage give the values of aligned ones; keys on a page outside the cache are left out and reported."""
    from ironpangu_b200.ops import decode as K

    g = torch.Generator(device="cuda").manual_seed(1)
    kv, hd, H, page, n = 2, 64, 16, 16, 90
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    kc, vc, q = rand(6, page, kv, hd), rand(6, page, kv, hd), rand(1, H * hd)
    off = lambda t: torch.empty(t.numel() + 4, dtype=BF16, device="cuda")[4:].view(t.shape).copy_(t)
    table = torch.arange(6, dtype=torch.int32, device="cuda").view(1, 6)
    pos, slots = torch.tensor([n - 1], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    how = dict(heads=H, kv_heads=kv, head_dim=hd, scale=0.125, keys_per_split=32, max_splits=4)
    a = K.gqa_decode_attention(q, kc, vc, pos, slots, table, **how)
    b = K.gqa_decode_attention(q, off(kc), off(vc), pos, slots, table, **how)
    torch.testing.assert_close(a.float(), b.float(), rtol=2 ** -7, atol=2e-4)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    table[0, 2] = 99
    c = K.gqa_decode_attention(q, kc, vc, pos, slots, table, status_ptr=status.data_ptr(), **how)
    keep = [i for i in range(n) if i // page != 2]
    ref = _reference(q.view(H, hd), kc.view(-1, kv, hd)[keep], vc.view(-1, kv, hd)[keep], 0.125).reshape(-1)
    torch.testing.assert_close(c[0].double(), ref, rtol=2 ** -8, atol=1e-4)
    assert int(status) == 4
