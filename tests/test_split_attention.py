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
        # a rounding to bf16 (at most 2^-8 of the value); f32 scores, weights and sums (2^-18 of values up to 5 is ample)
        torch.testing.assert_close(out[t].double(), ref, rtol=2 ** -8, atol=2e-5)
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


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("kps,splits,T", [(64, 8, 1), (128, 64, 1)])          # a cluster that merges by itself; parts that a second kernel merges
def test_weights_hold_24_bits(hd, kps, splits, T):
    """Values that cancel but for 2^-30 of them: what is left of the result is what the weights are off by, not the rounding of the result to bf16."""
    from ironpangu_b200.ops import decode as K

    g = torch.Generator(device="cuda").manual_seed(hd + splits)
    kv, group, page, n = 2, 2, 16, 40
    H = kv * group
    kc = torch.randn(3, page, kv, hd, generator=g, device="cuda").to(BF16)
    # query heads of a group are equal, so that one column of values cancels for both
    q = (torch.randn(T, kv, 1, hd, generator=g, device="cuda") * 0.5).to(BF16).expand(T, kv, group, hd).reshape(T, H * hd).contiguous()
    rows = kc.view(-1, kv, hd)[:n].double()
    w = torch.softmax(torch.einsum("gd,ngd->ng", q.view(T, kv, group, hd)[0, :, 0].double(), rows) * hd ** -0.5, 0)       # [n, kv]
    v = torch.randn(n, kv, hd, generator=g, device="cuda", dtype=torch.float64).to(BF16).double()
    left = torch.einsum("ng,ngd->gd", w[:n - 4], v[:n - 4])
    for i in range(n - 4, n):                      # every one of the last four takes away all but 2^-9 of what is left
        v[i] = (-left / w[i][:, None]).to(BF16).double()
        left = left + w[i][:, None] * v[i]
    vc = torch.zeros_like(kc)
    vc.view(-1, kv, hd)[:n] = v.to(BF16)
    table = torch.arange(3, dtype=torch.int32, device="cuda").view(1, 3)
    pos, slots = torch.full((T,), n - 1, dtype=torch.int32, device="cuda"), torch.zeros(T, dtype=torch.int32, device="cuda")
    out = K.gqa_decode_attention(q, kc, vc, pos, slots, table, heads=H, kv_heads=kv, head_dim=hd, scale=hd ** -0.5, keys_per_split=kps, max_splits=splits)
    of = torch.einsum("ng,ngd->gd", w, v.abs())
    off = ((out.view(T, kv, group, hd).double() - left[None, :, None]).abs() / of[None, :, None]).max()
    # the exponential (2^-21 of a weight) and scores up to 4 (2^-24 each) add up at random over 40 keys; 16 bits of a weight leave 2^-18
    assert float(off) < 2 ** -20, float(off)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("kps,splits", [(64, 8), (128, 64)])
def test_infinite_values_stay_infinite(hd, kps, splits):
    """An infinite value of a key gives an infinite result of its sign, whatever the key's weight is; the other columns are what they are without it."""
    from ironpangu_b200.ops import decode as K

    g = torch.Generator(device="cuda").manual_seed(hd + splits)
    kv, H, page, n = 1, 4, 16, 200
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    kc, vc, q = rand(13, page, kv, hd), rand(13, page, kv, hd), rand(1, H * hd) * 4
    kc.view(-1, hd)[7] = 0                          # equal scores: weights that bf16 holds exactly
    kc.view(-1, hd)[9] = -20 * q[0, :hd] / q[0, :hd].float().norm()       # a weight of next to nothing for the first head
    table = torch.arange(13, dtype=torch.int32, device="cuda").view(1, 13)
    pos, slots = torch.tensor([n - 1], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    how = dict(heads=H, kv_heads=kv, head_dim=hd, scale=hd ** -0.5, keys_per_split=kps, max_splits=splits)
    plain = K.gqa_decode_attention(q, kc, vc, pos, slots, table, **how).view(H, hd)
    for at in range(hd):
        vc.view(-1, hd)[[3, 7, 9, n - 1][at % 4], at] = float("-inf") if at % 3 == 0 else float("inf")
        if at % 8 == 7:
            vc.view(-1, hd)[:, at] = plain[0, at]   # a column without infinities
    out = K.gqa_decode_attention(q, kc, vc, pos, slots, table, **how).view(H, hd)
    for at in range(hd):
        want = plain[:, at] if at % 8 == 7 else torch.full((H,), float("-inf") if at % 3 == 0 else float("inf"), device="cuda")
        if at % 8 == 7:
            torch.testing.assert_close(out[:, at].float(), plain[0, at].float().expand(H), rtol=2 ** -7, atol=0)
        else:
            assert torch.equal(out[:, at].float(), want.float()), (at, out[:, at])


@pytest.mark.parametrize("hd,kv,group", [(128, 4, 4), (64, 4, 8), (128, 3, 1)])
@pytest.mark.parametrize("contexts", [[1], [129], [5000], [8191, 1, 4097], [65, 8000]])
def test_few_rows_of_long_contexts(hd, kv, group, contexts):
    """Up to 64 splits whose parts a second kernel merges: through the plain entry, and through that of windows with sinks and gates."""
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.ops import window_attn as WA

    g = torch.Generator(device="cuda").manual_seed(hd + kv + len(contexts))
    T, H, page, most = len(contexts), kv * group, 16, 512
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    kc, vc, q = rand(T * most, page, kv, hd), rand(T * most, page, kv, hd), rand(T, H * hd) * 2
    table = torch.randperm(T * most, generator=g, device="cuda").int().view(T, most)
    pos = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    slots = torch.arange(T, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.empty(T * H * 64 * (hd + 2), device="cuda")
    out = K.gqa_decode_attention(q, kc, vc, pos, slots, table, heads=H, kv_heads=kv, head_dim=hd, scale=hd ** -0.5, keys_per_split=128, max_splits=64, scratch=scratch,
                                 status_ptr=status.data_ptr())
    sink, gate, window = torch.randn(H, generator=g, device="cuda"), rand(T, H * hd), 4500
    seen = torch.empty(T, H * hd, dtype=BF16, device="cuda")
    WA.gqa_window(q, kc, vc, pos, slots, table, heads=H, window=window, scale=hd ** -0.5, splits=64, scratch=scratch, out=seen, sink=sink, gate=gate, gate_act="sigmoid",
                  status_ptr=status.data_ptr())
    for t, c in enumerate(contexts):
        k, v = (x[table[t].long()].reshape(-1, kv, hd)[:c].double().repeat_interleave(group, 1) for x in (kc, vc))
        s = torch.einsum("hd,nhd->hn", q[t].view(H, hd).double(), k) * hd ** -0.5
        torch.testing.assert_close(out[t].double(), torch.einsum("hn,nhd->hd", torch.softmax(s, -1), v).reshape(-1), rtol=2 ** -8, atol=2e-5)
        a = torch.softmax(torch.cat([s[:, max(0, c - window):], sink[:, None].double()], 1), -1)[:, :-1]
        want = torch.einsum("hn,nhd->hd", a, v[max(0, c - window):]).reshape(-1) * torch.sigmoid(gate[t].double())
        torch.testing.assert_close(seen[t].double(), want, rtol=2 ** -8, atol=2e-5)
    assert int(status) == 0


@pytest.mark.parametrize("kv,group,hd,n,kps,splits", [(4, 4, 128, 500, 128, 64), (4, 2, 128, 3000, 128, 64), (1, 8, 128, 4000, 128, 64), (4, 4, 64, 6000, 128, 64), (1, 4, 128, 6000, 4000, 2)])
def test_parts_are_f32_sums(kv, group, hd, n, kps, splits):
    """Maxima, sums and outputs of the splits as they lie in the scratch, before any rounding to bf16, against double precision."""
    from ironpangu_b200.ops import decode as K

    g = torch.Generator(device="cuda").manual_seed(n + hd)
    pages, H = (n + 15) // 16, kv * group
    kc, vc, q = (torch.randn(*s, generator=g, device="cuda").to(BF16) for s in ((pages, 16, kv, hd), (pages, 16, kv, hd), (1, H * hd)))
    q *= 2
    table, pos, slot = torch.arange(pages, dtype=torch.int32, device="cuda").view(1, -1), torch.tensor([n - 1], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.full((H * splits * (hd + 2),), float("nan"), device="cuda")
    K.gqa_decode_attention(q, kc, vc, pos, slot, table, heads=H, kv_heads=kv, head_dim=hd, scale=hd ** -0.5, keys_per_split=kps, max_splits=splits, scratch=scratch)
    most = min(splits, (296 + kv - 1) // kv)                                   # of one row
    parts = scratch[:H * most * (hd + 2)].view(H, most, hd + 2).double()
    parts = parts[:, ~parts[0, :, hd].isnan()]
    w = torch.exp(parts[..., hd] - parts[..., hd].max(-1, keepdim=True).values)
    out = (w[..., None] * parts[..., :hd]).sum(1) / (w * parts[..., hd + 1]).sum(-1)[:, None]
    k, v = (x.view(-1, kv, hd)[:n].double() for x in (kc, vc))
    s = torch.einsum("gjd,ngd->gjn", q.view(kv, group, hd).double(), k) * hd ** -0.5
    ref = torch.einsum("gjn,ngd->gjd", torch.softmax(s, -1), v).reshape(H, hd)
    # scores of up to 10 with a few roundings to 2^-24 of them, weights 2^-21 off at most: 4e-7 as f32 sums in any order are; where the tensor cores add up along a
    # whole row, cutting off, 6e-7 to 2e-6
    assert float((out - ref).norm() / ref.norm()) < 5.5e-7


# tiles of sixteen positions in pages that hold a multiple of them (16, 32, 48) and in others (24); windows that begin inside a tile; more than 32 tiles a warp (one
# split of 5000 keys); more CTAs than run at once, of rows of very different lengths (60 rows) and rows that are not there
@pytest.mark.parametrize("page,kv,group,hd,contexts,window,splits", [
    (16, 2, 4, 128, [5000], 0, 1), (32, 1, 8, 128, [5000, 40], 0, 1), (24, 2, 4, 128, [700, 33], 0, 8), (48, 2, 2, 64, [700, 48, 49], 0, 8),
    (16, 4, 4, 128, [1000, 65, 64, 17, 16, 3], 65, 8), (32, 2, 8, 64, [200, 31, 33], 33, 8), (16, 4, 4, 128, [17 * i + 1 if i % 7 else 0 for i in range(60)], 0, 64),
    (16, 4, 2, 64, [2000 - 30 * i for i in range(60)], 500, 8)])
def test_pages_windows_and_order(page, kv, group, hd, contexts, window, splits):
    from ironpangu_b200.ops.window_attn import gqa_window

    g = torch.Generator(device="cuda").manual_seed(page + hd + len(contexts))
    T, H = len(contexts), kv * group
    most = (max(contexts) + page - 1) // page
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    kc, vc, q = rand(T * most, page, kv, hd), rand(T * most, page, kv, hd), rand(T, H * hd)
    table = torch.randperm(T * most, generator=g, device="cuda").int().view(T, most)
    pos = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    slots = torch.arange(T, dtype=torch.int32, device="cuda")
    for t, c in enumerate(contexts):                     # what a row does not see must not count, whatever it holds
        if c and window and c > window:
            gone = (c - window) // page
            table[t, :gone] = -1
        rest = torch.arange(c, most * page, device="cuda")
        rows = table[t].long().clamp(min=0)[rest // page] * page + rest % page
        kc.view(-1, kv, hd)[rows] = float("nan")
        vc.view(-1, kv, hd)[rows] = float("nan")
    out = torch.full((T, H * hd), 7.0, dtype=BF16, device="cuda")
    scratch = torch.empty(T * H * 64 * (hd + 2), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    gqa_window(q, kc, vc, pos, slots, table, heads=H, window=window or max(contexts), scale=hd ** -0.5, splits=splits, scratch=scratch, out=out, status_ptr=status.data_ptr())
    for t, c in enumerate(contexts):
        if c == 0:
            assert bool((out[t] == 7).all())
            continue
        at = torch.arange(max(0, c - window) if window else 0, c, device="cuda")
        rows = table[t].long()[at // page] * page + at % page
        ref = _reference(q[t].view(H, hd), kc.view(-1, kv, hd)[rows], vc.view(-1, kv, hd)[rows], hd ** -0.5).reshape(-1)
        # a rounding to bf16 (at most 2^-8 of the value); f32 scores, weights and sums (2^-18 of values up to 5 is ample)
        torch.testing.assert_close(out[t].double(), ref, rtol=2 ** -8, atol=2e-5)
    assert int(status) == 0


def test_windows_take_the_parts_of_their_keys():
    """A row that sees a window of keys is shared as so many keys, wherever among sixteen positions its first one is: 33 parts of 128 keys, no 34th for keys ahead of the window."""
    from ironpangu_b200.ops.window_attn import gqa_window

    window, hd, group, splits, page = 33 * 128, 64, 4, 64, 16
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    for last in (6000, 6007, 6015):
        pages = last // page + 1
        kc, vc, q = rand(pages, page, 1, hd), rand(pages, page, 1, hd), rand(1, group * hd)
        table = torch.randperm(pages, generator=g, device="cuda").int()[None]
        pos, slots = torch.tensor([last], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        scratch = torch.full((group, splits, hd + 2), float("nan"), device="cuda")
        out = torch.empty(1, group * hd, dtype=BF16, device="cuda")
        gqa_window(q, kc, vc, pos, slots, table, heads=group, window=window, scale=hd ** -0.5, splits=splits, scratch=scratch, out=out)
        assert int(scratch.isfinite().all(-1)[0].sum()) == 33
        at = torch.arange(last + 1 - window, last + 1, device="cuda")
        rows = table[0].long()[at // page] * page + at % page
        ref = _reference(q.view(group, hd), kc.view(-1, 1, hd)[rows], vc.view(-1, 1, hd)[rows], hd ** -0.5).reshape(-1)
        # a rounding to bf16; f32 scores, weights and sums
        torch.testing.assert_close(out[0].double(), ref, rtol=2 ** -8, atol=2e-5)


@pytest.mark.parametrize("T,group,hd,window", [(31, 4, 128, 0), (32, 4, 128, 0), (33, 8, 64, 0), (33, 2, 128, 100), (34, 4, 128, 300), (37, 8, 128, 300)])
def test_about_as_many_clusters_as_run_at_once(T, group, hd, window):
    """Clusters of eight CTAs and of four, of eight warps and of four, over rows of one kv head (contexts to 600 keys)."""
    from ironpangu_b200.ops.window_attn import gqa_window

    g = torch.Generator(device="cuda").manual_seed(T + group)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)
    contexts = [1 + (37 * t) % 600 for t in range(T)]
    most = 38
    kc, vc, q = rand(T * most, 16, 1, hd), rand(T * most, 16, 1, hd), rand(T, group * hd)
    table = torch.randperm(T * most, generator=g, device="cuda").int().view(T, most)
    pos, slots = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda"), torch.arange(T, dtype=torch.int32, device="cuda")
    out = torch.empty(T, group * hd, dtype=BF16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    gqa_window(q, kc, vc, pos, slots, table, heads=group, window=window or 600, scale=hd ** -0.5, splits=((window or 600) + 63) // 64,
               scratch=torch.empty(T * group * 16 * (hd + 2), device="cuda"), out=out, status_ptr=status.data_ptr())
    for t, c in enumerate(contexts):
        at = torch.arange(max(0, c - window) if window else 0, c, device="cuda")
        rows = table[t].long()[at // 16] * 16 + at % 16
        ref = _reference(q[t].view(group, hd), kc.view(-1, 1, hd)[rows], vc.view(-1, 1, hd)[rows], hd ** -0.5).reshape(-1)
        # a rounding to bf16; f32 scores, weights and sums
        torch.testing.assert_close(out[t].double(), ref, rtol=2 ** -8, atol=2e-5)
    assert int(status) == 0


@pytest.mark.parametrize("T,kv,hd,longest", [(15, 1, 128, 300), (16, 1, 128, 300), (29, 1, 128, 300), (30, 1, 128, 300), (67, 1, 128, 300), (37, 2, 128, 300), (75, 1, 128, 300),
                                             (37, 4, 128, 300), (149, 1, 128, 300), (75, 2, 128, 1100), (74, 4, 128, 100), (99, 3, 128, 100), (31, 1, 64, 300), (65, 1, 64, 300),
                                             (67, 2, 64, 300), (149, 2, 64, 300)])
def test_splits_and_warps_by_rows(T, kv, hd, longest):
    """Both sides of where eight, four, two and one split of eight or four warps are taken, short and long rows of more than run at once."""
    test_pages_windows_and_order(16, kv, 4, hd, [1 + (37 * t) % longest for t in range(T - 1)] + [longest], 0, 64 if longest > 1024 else 8)
