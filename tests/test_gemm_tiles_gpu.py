"""The tile shapes of the projection GEMMs, at the row counts where the choice changes or a tile is ragged, and the
split-K projection + LayerNorm of small batches."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DT = {"f16": torch.float16, "bf16": torch.bfloat16}
ROUND = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}  # relative error of one rounding to 16 bits


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(0.7978845608028654 * (x + 0.044715 * x ** 3)))


# 768 columns: 64-, 128- and 256-column single-CTA tiles, 192- and 128-column pair tiles, whole waves + narrow tail;
# 2304 / 3072 columns: the same with more column tiles; 320 columns: only 64 divides
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("m,n,k", [(1, 768, 768), (129, 768, 3072), (1024, 768, 768), (2047, 768, 768), (4096, 768, 768),
                                   (5003, 768, 768), (8192, 768, 768), (7001, 768, 1024), (1025, 2304, 768),
                                   (2048, 2304, 768), (4353, 2304, 768), (1024, 3072, 768), (2049, 3072, 768),
                                   (5003, 3072, 768), (20481, 768, 768), (300, 320, 128), (300, 192, 64), (2305, 1024, 5120)])
@pytest.mark.parametrize("gelu", [False, True])
def test_gemm_tile_shapes(m, n, k, dtype, gelu):
    from raptor_t_b200 import capi, ops
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=gen).to(DT[dtype])
    w = (torch.randn(n, k, device="cuda", generator=gen) / k ** 0.5).to(DT[dtype])
    b = torch.randn(n, device="cuda", generator=gen).to(DT[dtype])
    guard = torch.full((m + 256, n), 7.0, device="cuda", dtype=DT[dtype])  # rows past the last must stay untouched
    out = ops.gemm(a, w, b, capi.RT_EPI_BIAS_GELU if gelu else capi.RT_EPI_BIAS, out=guard[:m])
    ref = a.double() @ w.double().t() + b.double()
    if gelu:
        ref = _gelu(ref)
    # one rounding of the result; the fp32 sum of k products and, with GELU, the approximate tanh (2^-10.9 absolute,
    # times x / 2) on top
    bound = ROUND[dtype] * ref.abs() + k * 2.0 ** -24 + (2.0 ** -10.9 * ref.abs() if gelu else 0.0) + 1e-5
    assert ((out.double() - ref).abs() <= bound).all()
    assert (guard[m:] == 7.0).all()
    ops.check_device()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("hidden,lens", [(768, [64]), (768, [128, 64]), (768, [512]), (768, [448, 576]), (768, [2048]),
                                         (768, [1984, 1408]), (1024, [64]), (1024, [512, 576])])
def test_split_k_projection_layernorm(hidden, lens, dtype):
    """FFN down + LayerNorm of a small batch (split-K parts summed by LayerNorm) against the unfused kernels of the
    same encoder: both round the output once; the unfused path rounds the projection once more."""
    from raptor_t_b200 import capi
    from raptor_t_b200.engine import Encoder
    import oracle
    cfg = dict(hidden=hidden, heads=hidden // 64, ffn=4 * hidden, layers=1, max_pos=4096, vocab=97)
    P = oracle.make_weights(oracle.EncoderConfig(**cfg), seed=5, nonzero_bias=True)
    enc = Encoder(capi.make_config(dtype=dtype, **cfg)).load_weights(P)
    ids = torch.randint(0, 97, (sum(lens),), device="cuda", dtype=torch.int32)
    split = enc.prepare(lens).forward_ids(ids).clone()
    again = enc.prepare(lens).forward_ids(ids).clone()
    assert torch.equal(split, again)
    enc.set_option("fuse_layernorm", 0)
    plain = enc.prepare(lens).forward_ids(ids).clone()
    # the projection is below 4 in magnitude here and LayerNorm divides by a deviation of order one
    bound = ROUND[dtype] * (2 * plain.double().abs() + 4)
    assert ((split.double() - plain.double()).abs() <= bound).all()
