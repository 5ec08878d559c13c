"""Work lists of a batch in one upload (short lists) or one per layer: forwards and per-operator calls agree, batches of both
kinds in turn through the same slots."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def test_one_upload_and_one_per_layer_in_turn():
    from raptor_t_b200 import capi, ops
    from raptor_t_b200.engine import Encoder
    cfg = dict(hidden=128, heads=2, ffn=256, layers=5, max_pos=4096, vocab=97)
    P = oracle.make_weights(oracle.EncoderConfig(**cfg), seed=3, nonzero_bias=True)
    enc = Encoder(capi.make_config(dtype="f16", **cfg)).load_weights(P)
    # 5 regions of about 2 KB, of 9 KB (both together in 64 KB), of 30 KB and more (a copy per layer)
    batches = [[64], [256, 1024], [4096, 832, 1024, 4096], [704] * 3, [1984] * 7]
    gen = torch.Generator(device="cuda").manual_seed(0)
    ids = [torch.randint(0, 97, (sum(b),), device="cuda", generator=gen, dtype=torch.int32) for b in batches]

    def by_operators(b, x):
        enc.prepare(b)
        h = torch.empty(sum(b), 128, device="cuda", dtype=torch.float16)
        enc.forward_ids(x, out=h)  # the tables of a forward, then the same layers one by one
        first = h.clone()
        enc.prepare(b)
        attn, mid = torch.empty_like(h), torch.empty(sum(b), 256, device="cuda", dtype=torch.float16)
        h.copy_(embed(b, x))
        for layer in range(5):
            enc.attention(layer, h, attn)
            enc.intermediate(layer, attn, mid)
            enc.output(layer, mid, attn, h)
        torch.cuda.synchronize()
        return first, h

    def embed(b, x):
        P32 = {k: v.cuda().float() for k, v in P.items()}
        pos = torch.cat([torch.arange(n, dtype=torch.int32, device="cuda") for n in b])
        return ops.embeddings(x, pos, torch.zeros_like(x), P32["embeddings.word_embeddings.weight"],
                              P32["embeddings.position_embeddings.weight"],
                              P32["embeddings.token_type_embeddings.weight"], P32["embeddings.LayerNorm.weight"],
                              P32["embeddings.LayerNorm.bias"], 1e-12, torch.float16)

    want = []
    for b, x in zip(batches, ids):
        first, single = by_operators(b, x)
        assert torch.equal(first, single), b
        want.append(first)
    order = [0, 2, 1, 0, 4, 3, 0, 0, 2, 0]
    got = [enc.prepare(batches[i]).forward_ids(ids[i]) for i in order]  # no synchronisation between batches
    for i, out in zip(order, got):
        assert torch.equal(out, want[i]), i
    ops.check_device()
    enc.close()
