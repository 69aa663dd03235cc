"""A row of a step has the bits that it has alone, whatever rows are beside it: steps of one to eight rows of the latent-attention + expert decoder."""
import pytest
import torch

pytestmark = pytest.mark.gpu
SEQ = [5, 77, 300, 12, 999, 41, 8, 650, 3, 17, 256, 533, 533, 588, 964]


def _run(chunks, fuse):
    from ironpangu_b200.models.mla_moe import MlaMoeConfig, MlaMoeDecoder, random_rank_weights
    from ironpangu_b200.parallel.fabric import Fabric

    cfg, fab = MlaMoeConfig.tiny(2), Fabric(0, 1)
    dec = MlaMoeDecoder(cfg, random_rank_weights(cfg, 0, 1, torch.device("cuda", 0), seed=0), fab, max_tokens=8, max_context=128, keep_logits=True)
    dec.fuse_override = fuse
    rows, logits, at = [], [], 0
    for n in chunks:
        dec.tokens[:n].copy_(torch.tensor(SEQ[at:at + n], dtype=torch.int32))
        dec.positions[:n].copy_(torch.arange(at, at + n, dtype=torch.int32))
        dec.slots[:n].zero_()
        dec.forward(n)
        rows.append(dec.x[:n].clone())
        logits.append(dec.logits[:n].clone())
        at += n
    assert fab.status() == 0
    fab.close()
    return torch.cat(rows), torch.cat(logits)


@pytest.mark.parametrize("chunks", [[8, 7], [3] * 5, [2, 6, 4, 3], [1, 8, 5, 1]])
def test_rows_are_those_of_steps_of_one(chunks):
    rows, logits = _run(chunks, False)
    alone, alone_logits = _run([1] * len(SEQ), False)
    assert torch.equal(rows, alone)
    # the head's f32 sums of steps of one and two and of more rows have orders of their own
    torch.testing.assert_close(logits, alone_logits, rtol=0, atol=2e-6 * float(alone_logits.abs().max()))
