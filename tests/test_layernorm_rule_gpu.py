"""Where a hidden-wide projection carries its LayerNorm: both sides of each line agree with the separate kernels."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks,fused", [(12, False), (13, True), (18, True), (19, True), (64, True), (65, True), (89, True), (90, True)])
def test_attention_output_on_both_sides_of_the_rule(blocks, fused):
    from raptor_t_b200 import capi, ops
    from raptor_t_b200.engine import Encoder
    cfg = dict(hidden=768, heads=12, ffn=3072, layers=1, max_pos=4096, vocab=97)
    P = oracle.make_weights(oracle.EncoderConfig(**cfg), seed=5, nonzero_bias=True)
    enc = Encoder(capi.make_config(dtype="f16", **cfg)).load_weights(P)
    T = 256 * blocks - 192  # the last row block is a single 64-token block
    lens = [1024] * (T // 1024) + ([T % 1024] if T % 1024 else [])
    enc.prepare(lens)
    assert enc.layernorm_in_projection()[0] == fused
    gen = torch.Generator(device="cuda").manual_seed(blocks)
    x = torch.randn(T, 768, device="cuda", generator=gen).half()
    out = enc.attention(0, x, torch.empty_like(x)).float()
    enc.set_option("fuse_layernorm", 0)
    apart = enc.attention(0, x, torch.empty_like(x)).float()
    ops.check_device()
    # one 16-bit rounding more before the LayerNorm on one side, and the result's on both: two units in the last place
    assert ((out - apart).abs() <= 2.0 ** -9 * apart.abs() + 2.0 ** -9).all(), (out - apart).abs().max().item()
    enc.close()


@pytest.mark.parametrize("blocks,fused", [(10, False), (11, True), (15, True), (16, False), (18, False), (19, True),
                                          (30, True), (31, False), (37, False), (38, True), (45, True), (46, False),
                                          (48, False), (49, True)])
def test_ffn_down_of_1024_columns_on_both_sides_of_the_rule(blocks, fused):
    from raptor_t_b200 import capi, ops
    from raptor_t_b200.engine import Encoder
    cfg = dict(hidden=1024, heads=16, ffn=4096, layers=1, max_pos=4096, vocab=97)
    P = oracle.make_weights(oracle.EncoderConfig(**cfg), seed=5, nonzero_bias=True)
    enc = Encoder(capi.make_config(dtype="f16", **cfg)).load_weights(P)
    T = 256 * blocks - 192
    enc.prepare([1024] * (T // 1024) + ([T % 1024] if T % 1024 else []))
    assert enc.layernorm_in_projection()[1] == fused
    gen = torch.Generator(device="cuda").manual_seed(blocks)
    f = torch.randn(T, 4096, device="cuda", generator=gen).half()
    x = torch.randn(T, 1024, device="cuda", generator=gen).half()
    out = enc.output(0, f, x, torch.empty_like(x)).float()
    enc.set_option("fuse_layernorm", 0)
    apart = enc.output(0, f, x, torch.empty_like(x)).float()
    ops.check_device()
    # the 16-bit sum before the LayerNorm of one side (at most a few standard deviations) and both results' rounding
    assert ((out - apart).abs() <= 2.0 ** -9 * apart.abs() + 2.0 ** -8).all(), (out - apart).abs().max().item()
    enc.close()
