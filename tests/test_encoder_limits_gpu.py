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


def _at(rows, cols, dtype, offset):
    """A tensor whose data starts `offset` elements behind a 256-byte boundary."""
    return torch.zeros(rows * cols + 64, device="cuda", dtype=dtype)[offset:offset + rows * cols].view(rows, cols)


# 128 tokens: split-K parts; 2816: both projections of the 1024-wide model carry their LayerNorm, as does the 768-wide
# attention output at 4096; 3840 tokens of 512: GEMM + LayerNorm
@pytest.mark.parametrize("hidden,lens", [(768, [128]), (768, [4096]), (1024, [128]), (1024, [2816]), (512, [128]),
                                         (512, [3840])])
def test_pointer_alignment_of_the_sublayers(hidden, lens):
    """16-byte aligned pointers are taken, except by the 768-wide FFN down (32); less is refused, never launched."""
    from raptor_t_b200 import capi, ops
    from raptor_t_b200.engine import _ptr
    enc = _encoder(hidden)
    T, dt = sum(lens), torch.float16
    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, hidden, device="cuda", generator=gen).to(dt)
    ffn = torch.randn(T, 4 * hidden, device="cuda", generator=gen).to(dt)
    enc.prepare(lens)
    st = torch.cuda.current_stream().cuda_stream
    attention = lambda o: capi.lib.rt_encoder_attention(enc._h, 0, _ptr(x), _ptr(o), st)  # noqa: E731
    output = lambda f, r, o: capi.lib.rt_encoder_output(enc._h, 0, _ptr(f), _ptr(r), _ptr(o), st)  # noqa: E731
    want = torch.empty_like(x), torch.empty_like(x)
    assert attention(want[0]) == capi.RT_OK and output(ffn, x, want[1]) == capi.RT_OK
    # both round the result once; the separate kernels round the projection (below 8 here) once more
    bound = lambda w: 2.0 ** -11 * (2 * w.double().abs() + 8)  # noqa: E731
    for offset in (2, 4, 8):
        o, r, f = _at(T, hidden, dt, offset), _at(T, hidden, dt, offset), _at(T, 4 * hidden, dt, offset)
        r.copy_(x)
        f.copy_(ffn)
        ok = offset == 8
        assert (attention(o) == capi.RT_OK) == ok
        if ok:
            assert ((o.double() - want[0].double()).abs() <= bound(want[0])).all()
        for args in ((f, x, o), (ffn, r, o), (ffn, x, o)):
            assert (output(*args) == capi.RT_OK) == (ok and hidden != 768)
        if ok and hidden != 768:
            assert ((o.double() - want[1].double()).abs() <= bound(want[1])).all()
    torch.cuda.synchronize()
    ops.check_device()
