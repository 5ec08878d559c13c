"""Projections of few rows: K split over a cluster of CTAs (8, 4 or 2 by the number of tiles), against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(M, N, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).to(dtype)
    return a, w, torch.randn(N, device="cuda", generator=g).to(dtype)


def _close(got, want, dtype, slack=0.0):
    # the result's rounding and K fp32 products of unit variance in total; slack: what an epilogue adds
    rel = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert ((got.double() - want).abs() <= rel * want.abs() + 2e-5 + slack).all(), (got.double() - want).abs().max().item()


# tiles * 8 <= 96, * 4 <= 128, * 2 <= 148, and one more than that; K blocks that do not divide evenly; rows around a tile's end;
# row blocks filled in part, on both sides of the lines for them
@pytest.mark.parametrize("N", [64, 768, 832, 2048, 2112, 2304, 2368, 3584, 3648, 4096, 4160, 4736, 4800])
@pytest.mark.parametrize("M,K", [(1, 512), (48, 640), (32, 2048), (64, 576), (95, 768), (96, 1024), (128, 768), (129, 1024),
                                 (191, 3072), (256, 832), (257, 768)])
def test_gemm_of_few_rows(M, N, K):
    from raptor_t_b200 import capi, ops
    dtype = torch.bfloat16 if (M + N // 64) % 2 else torch.float16
    a, w, bias = _inputs(M, N, K, dtype)
    acc = a.double() @ w.double().t()
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=dtype)
    _close(ops.gemm(a, w, None, capi.RT_EPI_NONE, out=out[:M]), acc, dtype)
    _close(ops.gemm(a, w, bias, capi.RT_EPI_BIAS, out=out[:M]), acc + bias.double(), dtype)
    # tanh.approx: 2^-10.987 relative, times half of the argument
    gelu = torch.nn.functional.gelu(acc + bias.double(), approximate="tanh")
    _close(ops.gemm(a, w, bias, capi.RT_EPI_BIAS_GELU, out=out[:M]), gelu, dtype,
           2.0 ** -11 * (acc + bias.double()).abs())
    res = torch.randn(M, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7)).to(dtype)
    _close(ops.gemm_residual(a, w, bias, res, out=out[:M]), acc + bias.double() + res.double(), dtype)
    assert (out[M] == 7.0).all()  # nothing behind the last row
    assert torch.equal(ops.gemm_residual(a, w, bias, res, out=res), out[:M])  # over the residual
    first = ops.gemm(a, w, bias, capi.RT_EPI_BIAS, out=torch.empty_like(out[:M])).clone()
    assert torch.equal(first, ops.gemm(a, w, bias, capi.RT_EPI_BIAS, out=torch.empty_like(out[:M])))
    ops.check_device()


@pytest.mark.parametrize("hidden,lens", [(768, [64]), (768, [128, 128]), (1024, [64, 128]), (512, [128, 64, 64])])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_layer_of_few_tokens_matches_the_oracle(hidden, lens, dtype):
    """QKV scatter, GELU and the fp32 sums that FFN down hands to its LayerNorm."""
    import oracle
    from raptor_t_b200 import capi, ops
    from raptor_t_b200.engine import Encoder
    cfg = dict(hidden=hidden, heads=hidden // 64, ffn=4 * hidden, layers=1, max_pos=4096, vocab=97)
    ocfg = oracle.EncoderConfig(**cfg)
    P = oracle.make_weights(ocfg, seed=5, nonzero_bias=True)
    enc = Encoder(capi.make_config(dtype=dtype, **cfg)).load_weights(P)
    gen = torch.Generator().manual_seed(1)
    seqs = [torch.randint(0, 97, (n,), generator=gen, dtype=torch.int32) for n in lens]
    enc.prepare(lens)
    out = enc.forward_ids(torch.cat(seqs).cuda()).float().cpu()
    ops.check_device()
    err = (out - oracle.encoder_ref(seqs, P, ocfg)).abs()
    bound = (2e-2, 2e-3) if dtype == "f16" else (1.6e-1, 1.6e-2)  # the path's bounds at 11 and 8 bits
    assert err.max().item() < bound[0] and err.mean().item() < bound[1], (err.max().item(), err.mean().item())
    enc.close()
