"""The encoder object at the edges of its memory: a batch that does not fit the device."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _encoder(hidden, layers=1, dtype="f16", ffn=None):
    from raptor_t_b200 import capi
    from raptor_t_b200.engine import Encoder
    cfg = dict(hidden=hidden, heads=hidden // 64, ffn=ffn or 4 * hidden, layers=layers, max_pos=4096, vocab=97)
    P = oracle.make_weights(oracle.EncoderConfig(**cfg), seed=5, nonzero_bias=True)
    return Encoder(capi.make_config(dtype=dtype, **cfg)).load_weights(P)


def test_batch_that_does_not_fit_leaves_the_encoder_usable():
    """The allocation for it fails and the next, smaller batch has memory of its own again."""
    from raptor_t_b200 import ops
    enc = _encoder(128, layers=2)
    ids = torch.randint(0, 97, (832,), device="cuda", dtype=torch.int32)
    want = enc.prepare([832]).forward_ids(ids).clone()
    per_token = 2 * (9 * 128 + 512)  # 16-bit scratch of one token
    too_many = int(1.2 * torch.cuda.mem_get_info()[1] / per_token / 4096)
    with pytest.raises(Exception, match="memory"):
        enc.prepare([4096] * too_many)
    torch.cuda.synchronize()
    small = torch.empty(1 << 22, device="cuda").fill_(3.0)  # takes what the failed batch gave back
    assert torch.equal(enc.prepare([832]).forward_ids(ids), want)
    assert (small == 3.0).all()
    ops.check_device()
