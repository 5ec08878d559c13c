"""Residual + bias + LayerNorm where a warp walks several rows: fewer rows than warps, one more than a whole round of the
grid, ragged ends, every row width's vector count, in place and without bias and residual."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [64, 128, 520, 768, 1024, 1536, 2048])
@pytest.mark.parametrize("rows", [1, 7, 2369, 7105, 14209])
def test_rows_match_float64(rows, hidden):
    from raptor_t_b200 import ops
    dtype = torch.bfloat16 if (rows + hidden // 8) % 2 else torch.float16
    gen = torch.Generator(device="cuda").manual_seed(rows + hidden)
    x, res = (torch.randn(rows, hidden, device="cuda", generator=gen).to(dtype) for _ in range(2))
    bias, beta = ((torch.randn(hidden, device="cuda", generator=gen) * 0.1).to(dtype) for _ in range(2))
    gamma = (1.0 + 0.1 * torch.randn(hidden, device="cuda", generator=gen)).to(dtype)
    # the result's rounding (half a unit in the last place) and fp32 sums of up to 2048 terms far below it
    rel = 2.0 ** (-8 if dtype == torch.bfloat16 else -11) + 1e-5

    def check(got, total):
        want = torch.nn.functional.layer_norm(total, (hidden,), gamma.double(), beta.double(), 1e-12)
        assert ((got.double() - want).abs() <= rel * want.abs() + 1e-5).all()

    total = x.double() + bias.double() + res.double()
    check(ops.bias_residual_layernorm(x, bias, res, gamma, beta, 1e-12, out=torch.empty_like(x)), total)
    check(ops.bias_residual_layernorm(x.clone(), None, None, gamma, beta, 1e-12), x.double())
    check(ops.bias_residual_layernorm(x, bias, res, gamma, beta, 1e-12, out=res), total)
    ops.check_device()
