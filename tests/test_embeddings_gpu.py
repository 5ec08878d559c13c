"""Embedding gather + LayerNorm at row widths that do not fill a warp's pieces, and with unaligned parameters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens,hidden", [(1, 8), (7, 136), (4097, 128), (65, 264), (6001, 768), (33, 1000), (5, 1024)])
@pytest.mark.parametrize("offset", [0, 1])
def test_embeddings(tokens, hidden, dtype, offset):
    from raptor_t_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    word, pos, typ = (torch.randn(n, hidden, device="cuda", generator=gen) for n in (97, 64, 2))
    gamma = torch.randn(hidden + 1, device="cuda", generator=gen)[offset:offset + hidden]  # offset 1: 4-byte aligned only
    beta = torch.randn(hidden + 1, device="cuda", generator=gen)[offset:offset + hidden]
    ids, pids, tids = (torch.randint(0, n, (tokens,), device="cuda", generator=gen, dtype=torch.int32) for n in (97, 64, 2))
    out = ops.embeddings(ids, pids, tids, word, pos, typ, gamma, beta, 1e-12, dtype)
    x = word.double()[ids.long()] + typ.double()[tids.long()] + pos.double()[pids.long()]
    ref = torch.nn.functional.layer_norm(x, (hidden,), gamma.double(), beta.double(), 1e-12)
    # one rounding of the result to 16 bits, and fp32 statistics
    bound = (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * ref.abs() + 1e-5 * (1 + gamma.double().abs())
    assert ((out.double() - ref).abs() <= bound * 1.01).all()
