"""Parameters replaced between forwards: the copies are done when the call returns, whatever stream the forwards before and
after it run on."""
import ctypes as C

import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

CFG = dict(hidden=128, heads=2, ffn=256, layers=2, max_pos=4096, vocab=97)
LENS = [64, 128]


def _encoder(seed):
    from raptor_t_b200 import capi
    from raptor_t_b200.engine import Encoder
    P = oracle.make_weights(oracle.EncoderConfig(**CFG), seed=seed, nonzero_bias=True)
    return Encoder(capi.make_config(dtype="f16", **CFG)).load_weights(P), P


def _layer_tensors(P, layer):
    pre = f"encoder.layer.{layer}."
    qkv = ["attention.self.query", "attention.self.key", "attention.self.value"]
    ts = [torch.cat([P[pre + n + "." + k] for n in qkv]) for k in ("weight", "bias")]
    for n in ("attention.output.dense", "attention.output.LayerNorm", "intermediate.dense", "output.dense",
              "output.LayerNorm"):
        ts += [P[pre + n + ".weight"], P[pre + n + ".bias"]]
    return [t.cuda().half().contiguous() for t in ts]


def _set(enc, P):
    """As a C caller does: nothing waits but the entry points themselves."""
    from raptor_t_b200.capi import check, lib
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    layers = [_layer_tensors(P, i) for i in range(CFG["layers"])]
    e = "embeddings."
    emb = [P[e + n].cuda().float().contiguous() for n in
           ("word_embeddings.weight", "position_embeddings.weight", "token_type_embeddings.weight", "LayerNorm.weight",
            "LayerNorm.bias")]
    torch.cuda.synchronize()
    calls = [lambda i=i, ts=ts: check(lib.rt_encoder_set_layer(enc._h, i, i, 0, *map(p, ts))) for i, ts in enumerate(layers)]
    calls.append(lambda: check(lib.rt_encoder_set_embeddings(enc._h, *map(p, emb))))
    for call in calls:
        torch.cuda._sleep(20_000_000)  # the copies' stream is busy for some ms
        call()
        assert torch.cuda.default_stream().query()


def test_forwards_before_and_after_have_their_own_parameters():
    from raptor_t_b200 import ops
    ids = torch.randint(0, 97, (sum(LENS),), generator=torch.Generator().manual_seed(0), dtype=torch.int32)
    (a, _), (b, P) = _encoder(3), _encoder(4)
    want_a, want_b = (e.prepare(LENS).forward_ids(ids.cuda()).clone() for e in (a, b))
    torch.cuda.synchronize()
    side, dev = torch.cuda.Stream(), ids.cuda()
    before = torch.empty_like(want_a)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        a.prepare(LENS).forward_ids(dev, out=before)
    _set(a, P)
    host = torch.empty(want_b.shape, dtype=want_b.dtype).pin_memory()
    a.forward_host(LENS, ids.pin_memory(), host)  # the object's own stream
    torch.cuda.synchronize()
    assert torch.equal(before, want_a)
    assert torch.equal(host, want_b.cpu())
    ops.check_device()
    a.close()
    b.close()
