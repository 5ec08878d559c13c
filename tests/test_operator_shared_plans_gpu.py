"""Operator classes of several live models: layers with the same block lists share one work list per batch."""
import gc

import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _model(raptor_t, heads, seed, async_=True):
    from raptor_t_b200.modeling_bert import BertModelNoPooler
    cfg = oracle.EncoderConfig(hidden=64 * heads, heads=heads, ffn=256, layers=2, max_pos=4096, vocab=97)
    P = oracle.make_weights(cfg, seed=seed, nonzero_bias=True)
    return cfg, P, BertModelNoPooler.from_weights(P, cfg.hidden, heads, cfg.ffn, cfg.layers, torch.float16, async_,
                                                  backend=raptor_t)


# short sequences only (one list for all layers), random blocks, both, and a list that is cut
@pytest.mark.parametrize("lens", [[256, 704], [832, 1024], [4096], [320, 1984, 64 * 11]])
def test_models_alive_together_match_the_oracle(lens):
    from raptor_t_b200 import compiled, metadata, ops
    raptor_t = compiled.load()
    models = [_model(raptor_t, 2, 3), _model(raptor_t, 2, 4), _model(raptor_t, 3, 5), _model(raptor_t, 2, 6, False)]
    md = raptor_t.MetaData()
    prefix, total, _, _ = metadata.generate_data_metainfo(lens, 64, 160, 2) if min(lens) >= 256 else \
        ([sum(lens[:i]) // 64 for i in range(len(lens) + 1)], 0, None, None)
    T = sum(lens)
    ids = torch.randint(0, 97, (T,), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
    pos = torch.cat([torch.arange(n, dtype=torch.int32) for n in lens]).cuda()
    prefix_dev = torch.tensor(prefix, dtype=torch.int32, device="cuda")

    def forward(m):
        return m(ids.cuda(), T, 160, prefix, prefix_dev, position_ids=pos, test_info={})[0]

    def check(cfg, P, m):
        ref = oracle.encoder_ref(list(ids.split(lens)), P, cfg)
        err = (forward(m).float().cpu() - ref).abs()
        # fp16 against the fp32 oracle, the bound of the path
        assert err.max().item() < 2e-2 and err.mean().item() < 2e-3, (err.max().item(), err.mean().item())

    md.update_meta_data(T, prefix[-1] + 1, total, prefix)
    for cfg, P, m in models + models[:1]:
        check(cfg, P, m)
    # the plan outlives the model that came first, also before its task has been joined
    md.update_meta_data(T, prefix[-1] + 1, total, prefix)
    m = None
    models.pop(0)
    gc.collect()
    for cfg, P, m in models:
        check(cfg, P, m)
    md.terminate_thread()
    ops.check_device()


def test_models_on_two_streams_share_partial_results():
    """A list that is cut leaves its partial results in the plan, which both models now share: forwards of the two on two
    streams, issued without any synchronisation, layer by layer in turn, come out as alone."""
    from raptor_t_b200 import compiled, metadata, ops
    raptor_t = compiled.load()
    models = [_model(raptor_t, 2, seed)[2] for seed in (3, 4)]
    md = raptor_t.MetaData()
    lens = [4096]
    prefix, total, _, _ = metadata.generate_data_metainfo(lens, 64, 160, 2)
    T = sum(lens)
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = [torch.randn(T, 128, device="cuda", generator=gen).half() for _ in models]
    mask = None
    prefix_dev = torch.tensor(prefix, dtype=torch.int32, device="cuda")
    md.update_meta_data(T, prefix[-1] + 1, total, prefix)

    def attention(m, layer, src, dst):
        m.encoder.layer[layer].attention(src, mask, dst, prefix, prefix_dev, None, None, 160, {})

    want = []
    for m, src in zip(models, x):
        a, b = torch.empty_like(src), torch.empty_like(src)
        attention(m, 0, src, a)
        attention(m, 1, a, b)
        want.append(b)
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[(torch.empty_like(src), torch.empty_like(src)) for src in x] for _ in range(6)]
    torch.cuda.synchronize()
    for rep in got:
        for layer in (0, 1):
            for m, s, src, (a, b) in zip(models, streams, x, rep):
                with torch.cuda.stream(s):
                    attention(m, layer, src if layer == 0 else a, a if layer == 0 else b)
    torch.cuda.synchronize()
    for rep in got:
        for w, (_, b) in zip(want, rep):
            assert torch.equal(b, w)
    md.terminate_thread()
    ops.check_device()
