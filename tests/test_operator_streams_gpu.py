"""The compiled operator classes in a serving loop: batches of changing lengths, metadata uploaded on one stream and the
model run on another, plans of earlier batches given back while their kernels may still run."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_streams", [False, True])
def test_batches_in_a_loop_match_single_batches(two_streams):
    from raptor_t_b200 import compiled, metadata, ops
    from raptor_t_b200.modeling_bert import BertModelNoPooler
    raptor_t = compiled.load()
    cfg = oracle.EncoderConfig(hidden=128, heads=2, ffn=256, layers=2, max_pos=4096, vocab=97)
    P = oracle.make_weights(cfg, seed=3, nonzero_bias=True)
    model = BertModelNoPooler.from_weights(P, cfg.hidden, cfg.heads, cfg.ffn, cfg.layers, torch.float16, True,
                                           backend=raptor_t)
    md = raptor_t.MetaData()
    batches = []
    for i, lens in enumerate([[832, 1024], [256], [4096, 512, 1984], [1024] * 5, [320, 832]]):
        prefix, total, part_off, part_ids = metadata.generate_data_metainfo(lens, 64, 160, cfg.heads)
        T = sum(lens)
        gen = torch.Generator(device="cuda").manual_seed(i)
        batches.append(dict(T=T, prefix=prefix, total=total,
                            ids=torch.randint(0, 97, (T,), device="cuda", generator=gen, dtype=torch.int32),
                            pos=torch.cat([torch.arange(n, dtype=torch.int32, device="cuda") for n in lens]),
                            prefix_dev=torch.tensor(prefix, dtype=torch.int32, device="cuda"),
                            off=torch.from_numpy(part_off).cuda(), part=torch.from_numpy(part_ids).cuda()))
    torch.cuda.synchronize()

    def step(b, stream):
        md.update_meta_data(b["T"], b["prefix"][-1] + 1, b["total"], b["prefix"])
        with torch.cuda.stream(stream):
            return model(b["ids"], b["T"], 160, b["prefix"], b["prefix_dev"], b["off"], b["part"],
                         position_ids=b["pos"], test_info={})[0]

    default = torch.cuda.default_stream()
    want = []
    for b in batches:
        want.append(step(b, default).clone())
        torch.cuda.synchronize()
    other = torch.cuda.Stream() if two_streams else default
    got = [step(b, other) for _ in range(3) for b in batches]  # no synchronisation between batches
    torch.cuda.synchronize()
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % len(batches)]), i
    md.terminate_thread()
    ops.check_device()


def test_update_meta_data_refuses_a_capturing_stream():
    from raptor_t_b200 import compiled
    md = compiled.load().MetaData()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        with pytest.raises(RuntimeError, match="captured"):
            md.update_meta_data(1024, 17, 100, [0, 16])
