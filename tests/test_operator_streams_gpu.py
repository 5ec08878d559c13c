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


def _model_and_batches(heads, lens_of_batches):
    from raptor_t_b200 import compiled, metadata
    from raptor_t_b200.modeling_bert import BertModelNoPooler
    raptor_t = compiled.load()
    cfg = oracle.EncoderConfig(hidden=64 * heads, heads=heads, ffn=256, layers=2, max_pos=4096, vocab=97)
    P = oracle.make_weights(cfg, seed=3, nonzero_bias=True)
    model = BertModelNoPooler.from_weights(P, cfg.hidden, cfg.heads, cfg.ffn, cfg.layers, torch.float16, True,
                                           backend=raptor_t)
    md = raptor_t.MetaData()
    batches = []
    for i, lens in enumerate(lens_of_batches):
        prefix, total, _, _ = metadata.generate_data_metainfo(lens, 64, 160, cfg.heads)
        gen = torch.Generator(device="cuda").manual_seed(i)
        batches.append(dict(T=sum(lens), prefix=prefix, total=total,
                            ids=torch.randint(0, 97, (sum(lens),), device="cuda", generator=gen, dtype=torch.int32),
                            pos=torch.cat([torch.arange(n, dtype=torch.int32, device="cuda") for n in lens]),
                            prefix_dev=torch.tensor(prefix, dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()

    def update(b):
        md.update_meta_data(b["T"], b["prefix"][-1] + 1, b["total"], b["prefix"])

    def forward(b):
        return model(b["ids"], b["T"], 160, b["prefix"], b["prefix_dev"], position_ids=b["pos"], test_info={})[0]

    return md, batches, update, forward


def _wanted(batches, update, forward):
    want = []
    for b in batches:
        update(b)
        want.append(forward(b).clone())
        torch.cuda.synchronize()
    return want


def test_batches_on_alternating_streams():
    """The operator objects share scratch: a batch on another stream comes behind the one before it, also where the
    scratch grows there, and nobody synchronises."""
    from raptor_t_b200 import ops
    md, batches, update, forward = _model_and_batches(3, [[256], [512, 1984], [4096, 1024], [320], [1024] * 7])
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got, done = [], []
    for i in range(4 * len(batches)):  # 5 batches, 2 streams: every batch comes on both
        b, s = batches[i % len(batches)], streams[i % 2]
        update(b)
        with torch.cuda.stream(s):
            if i % 4 == 1:
                torch.cuda._sleep(20_000_000)  # this stream is late: the next batch must not overtake it
            got.append(forward(b))
            done.append(s.record_event())
    done[-1].synchronize()
    assert all(e.query() for e in done)
    torch.cuda.synchronize()
    for i, w in enumerate(_wanted(batches, update, forward)):
        for out in got[i::len(batches)]:
            assert torch.equal(out, w), i
    md.terminate_thread()
    ops.check_device()


def test_captured_forward_replays():
    """A warm model captures into a graph on another stream than the metadata was uploaded on, and the next batch's
    metadata waits for replays in flight."""
    from raptor_t_b200 import ops
    md, batches, update, forward = _model_and_batches(2, [[832, 1024], [4096, 512]])
    want = _wanted(batches, update, forward)
    b = batches[0]
    update(b)
    forward(b)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = forward(b)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0])
    b["ids"].copy_(b["ids"].flip(0))
    flipped = forward(b).clone()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, flipped) and not torch.equal(flipped, want[0])
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
        g.replay()
        done = s.record_event()
    update(batches[1])
    assert done.query()
    assert torch.equal(forward(batches[1]), want[1])
    torch.cuda.synchronize()
    assert torch.equal(out, flipped)
    md.terminate_thread()
    ops.check_device()


def test_stream_destroyed_between_batches():
    """Nothing of a batch on a caller's own stream is touched through that stream once the caller has waited for it and
    destroyed it."""
    import ctypes
    from raptor_t_b200 import ops
    md, batches, update, forward = _model_and_batches(2, [[4096, 512], [832, 1024]])
    want = _wanted(batches, update, forward)
    rt = torch.cuda.cudart()
    for i in range(4):
        handle = ctypes.c_ulonglong(0)
        assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
        own = torch.cuda.ExternalStream(handle.value)
        update(batches[i % 2])
        with torch.cuda.stream(own):
            out = forward(batches[i % 2])
        own.synchronize()
        assert int(rt.cudaStreamDestroy(handle.value)) == 0
        assert torch.equal(out, want[i % 2])
    update(batches[1])
    assert torch.equal(forward(batches[1]), want[1])
    md.terminate_thread()
    ops.check_device()
