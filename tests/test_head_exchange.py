"""The greedy head between ranks, and what it refuses. The other rank's candidates and its flag are in place before the launch, so nothing is waited for."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("kept", [False, True])
@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 8])
def test_candidates_lie_where_every_form_of_the_head_looks(T, kept):
    """Slot 8 * rank + token, whether a rank keeps its logits (a product and a selection) or not: ranks may differ in that."""
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.parallel.fabric import Fabric, _CudaBuffer

    g = torch.Generator(device="cuda").manual_seed(T)
    fab = Fabric(0, 2, silent_peers=True, spin_limit=2000)
    mine, theirs = (torch.as_tensor(_CudaBuffer(p, fab.bytes), device="cuda") for p in (fab.base, fab._silent[0]))
    half = fab.data_half_bytes                      # the first call's parity is 1
    slots = lambda block: block[half:half + 2 * 8 * 8].view(2, 8, 8)
    value, index = lambda s: s[..., :4].view(torch.float32)[..., 0], lambda s: s[..., 4:].view(torch.int32)[..., 0]
    at = slots(mine)[1]
    best = torch.tensor([1e9 if t % 2 else -1e9 for t in range(8)], device="cuda")
    at[:, :4].view(torch.float32)[:, 0] = best
    at[:, 4:].view(torch.int32)[:, 0] = torch.arange(5000, 5008, dtype=torch.int32, device="cuda")
    flag = fab._off_flags + (fab.flag_half_words + 1) * 8
    mine[flag:flag + 8].view(torch.int64)[0] = 1
    x, w = torch.randn(T, 256, generator=g, device="cuda").to(BF16), torch.randn(1000, 256, generator=g, device="cuda").to(BF16)
    ref = x.float() @ w.float().T
    logits = torch.empty(T, 1000, device="cuda") if kept else None
    ids = K.lm_head_argmax(x, w, fab, vocab_offset=100, logits=logits)
    own = ref.argmax(-1) + 100
    assert ids.tolist() == [5000 + t if t % 2 else int(own[t]) for t in range(T)]
    sent = slots(theirs)[0]
    assert index(sent)[:T].tolist() == own.tolist()
    torch.testing.assert_close(value(sent)[:T], ref.max(-1).values, rtol=1e-4, atol=1e-3)
    assert fab.status() == 0
    fab.close()


@pytest.mark.parametrize("T", [3, 4, 8])
def test_room_for_the_maxima_is_asked_for_in_either_form(T):
    """Logits kept or not, the same partial buffer is too small (and the same is large enough)."""
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.parallel.fabric import Fabric

    fab = Fabric(0, 1)
    V, D = 1000, 64
    x, w = torch.randn(T, D, device="cuda").to(BF16), torch.randn(V, D, device="cuda").to(BF16)
    need = (V + 31) // 32 * 4 * 8 if T <= 4 else (V + 15) // 16 * 8 * 8
    ids = {}
    for logits in (None, torch.empty(T, V, device="cuda")):
        with pytest.raises(RuntimeError):
            K.lm_head_argmax(x, w, fab, norm_w=torch.ones(D, device="cuda", dtype=BF16), logits=logits, partial=torch.empty(need // 4 - 2, device="cuda"))
        ids[logits is None] = K.lm_head_argmax(x, w, fab, norm_w=torch.ones(D, device="cuda", dtype=BF16), logits=logits, partial=torch.empty(need // 4, device="cuda"))
    ref = torch.nn.functional.rms_norm(x.float(), (D,), eps=1e-5).to(BF16).float() @ w.float().T
    for i in ids.values():                          # any of the nearly largest: both forms add up in an order of their own
        assert bool((ref.gather(1, i.long()[:, None])[:, 0] >= ref.max(-1).values - 1e-2).all())
    assert fab.status() == 0
    fab.close()
