"""FFN down + LayerNorm of small batches, split along K: the LayerNorm that sums the fp32 parts, one CTA or one warp per row,
on both sides of the lines between them, against float64."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,dtype", [(128, "bf16"), (256, "f16"), (384, "bf16"), (512, "f16"), (640, "bf16"), (768, "f16"),
                                          (768, "bf16"), (896, "f16"), (1024, "bf16")])
def test_ffn_down_of_small_batches(hidden, dtype):
    from raptor_t_b200 import capi, ops
    from raptor_t_b200.engine import Encoder
    ffn = max(4 * hidden, 2048)  # shorter sums are not split
    cfg = dict(hidden=hidden, heads=hidden // 64, ffn=ffn, layers=1, max_pos=4096, vocab=97)
    P = oracle.make_weights(oracle.EncoderConfig(**cfg), seed=5, nonzero_bias=True)
    enc = Encoder(capi.make_config(dtype=dtype, **cfg)).load_weights(P)
    td = torch.float16 if dtype == "f16" else torch.bfloat16
    pre = "encoder.layer.0.output."
    W = {k: P[pre + k].cuda().to(td).double() for k in ("dense.weight", "dense.bias", "LayerNorm.weight", "LayerNorm.bias")}
    split = 0
    for rows in (64, 256, 320, 512, 576, 896, 960, 1024, 1472, 1536, 1600, 2048, 2112, 2304, 2368, 5888, 6144):
        enc.prepare([rows] if rows <= 4096 and rows != 768 else [rows // 2] * 2)
        split += enc.get_option("ffn_down_parts") > 0
        gen = torch.Generator(device="cuda").manual_seed(rows)
        f = torch.randn(rows, ffn, device="cuda", generator=gen).to(td)
        x = torch.randn(rows, hidden, device="cuda", generator=gen).to(td)
        out = enc.output(0, f, x, torch.empty_like(x))
        want = torch.nn.functional.layer_norm(f.double() @ W["dense.weight"].t() + W["dense.bias"] + x.double(), (hidden,),
                                              W["LayerNorm.weight"], W["LayerNorm.bias"], 1e-12)
        # the result's rounding; where the sums are rounded to 16 bits on the way (no parts), that of a row's values, too
        eps = 2.0 ** (-11 if dtype == "f16" else -8)
        slack = 2e-5 if enc.get_option("ffn_down_parts") else 6 * eps
        assert ((out.double() - want).abs() <= eps * want.abs() + slack).all(), rows
        again = enc.output(0, f, x, x)  # in place of the residual, too
        assert torch.equal(again, out), rows
    assert split >= 5
    ops.check_device()
    enc.close()
