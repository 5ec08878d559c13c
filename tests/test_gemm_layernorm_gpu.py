"""Projection + LayerNorm in one kernel: parameters that the kernel before has just written, and rows whose mean is far
above their deviation."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DT = {"f16": torch.float16, "bf16": torch.bfloat16}
ROUND = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}  # relative error of one rounding to 16 bits
SHAPES = [(100, 768, 768), (5003, 768, 768), (300, 1024, 1024)]  # single-CTA clusters, clusters of 3 and of 4 pairs


def _operands(m, n, k, dtype):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=gen).to(DT[dtype])
    w = (torch.randn(n, k, device="cuda", generator=gen) / k ** 0.5).to(DT[dtype])
    return gen, a, w, torch.randn(m, n, device="cuda", generator=gen).to(DT[dtype])


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_parameters_written_by_the_kernel_before(m, n, k, dtype):
    """bias, gamma and beta are the last rows of a tensor that bias + GELU, which lets the next kernel start early, has
    just overwritten: the same bits as with parameters that are long there."""
    from raptor_t_b200 import ops
    gen, a, w, res = _operands(m, n, k, dtype)
    rows = torch.randn(40000, n, device="cuda", generator=gen).to(DT[dtype])
    zero = torch.zeros(n, device="cuda", dtype=DT[dtype])
    par = ops.bias_gelu_(rows.clone(), zero)
    torch.cuda.synchronize()
    want = ops.gemm_bias_residual_layernorm(a, w, par[-1], res, par[-2], par[-3], 1e-12)
    torch.cuda.synchronize()
    out = torch.empty_like(want)
    for _ in range(5):
        fresh = rows.clone()
        torch.cuda.synchronize()
        ops.bias_gelu_(fresh, zero)
        ops.gemm_bias_residual_layernorm(a, w, fresh[-1], res, fresh[-2], fresh[-3], 1e-12, out=out)
        assert torch.equal(out, want)
    ops.check_device()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_rows_with_a_mean_far_above_their_deviation(m, n, k, dtype):
    """A bias of 1536 under a deviation of about 2.7: the mean of the squares minus the squared mean would leave 4 bits."""
    from raptor_t_b200 import ops
    mean = 1536.0
    gen, a, w, _ = _operands(m, n, k, dtype)
    res = torch.randint(-4, 5, (m, n), device="cuda", generator=gen).to(DT[dtype])
    bias = torch.full((n,), mean, device="cuda", dtype=DT[dtype])
    gamma, beta = (torch.randn(n, device="cuda", generator=gen).to(DT[dtype]) for _ in range(2))
    out = ops.gemm_bias_residual_layernorm(a, w, bias, res, gamma, beta, 1e-12)
    x = a.double() @ w.double().t() + bias.double() + res.double()
    ref = torch.nn.functional.layer_norm(x, (n,), gamma.double(), beta.double(), 1e-12)
    # one rounding of the result; x itself and the row's mean in fp32: two additions of 2^-24 |mean| each, and a sum of
    # 64 packed pairs and 2 n / 128 parts, against a deviation above 2.4 (once through the mean, once through 1/sigma,
    # which an error of the mean enters squared); the sum of k products of magnitude below 16
    shift = ((64 + n // 64 + 4) * mean + k * 16.0) * 2.0 ** -24 / 2.4
    bound = ROUND[dtype] * ref.abs() + shift * gamma.double().abs() + 1e-5
    assert ((out.double() - ref).abs() <= bound * 1.01).all()
    ops.check_device()
