"""The work that this encoder is used for, as timed cases over its public entry points.

Kinds of a case:

* ``encoder``    one batch through ``Encoder.prepare`` + ``Encoder.forward_ids`` (ids on the device): the serving call.
* ``host``       one batch through ``Encoder.forward_host`` (pinned ids in, hidden states out in pinned memory).
* ``operators``  one batch through the operator classes (compiled module ``raptor_t``) and the Python model layer on
                 them: ``MetaData.update_meta_data`` + ``BertModelNoPooler``.
* ``attention``  the block-sparse attention alone, with its plan in hand.
* ``projection`` one projection GEMM with its epilogue.
* ``layernorm``  residual + bias + LayerNorm over packed rows.

Model shapes are those of the repository's benchmark: ``base`` (12 layers, hidden 768), ``band`` (base with a 512-token
window instead of the random blocks) and ``large`` (24 layers, hidden 1024).  Batches are packed without padding;
sequence lengths are multiples of the 64-token block and ragged.
"""
import math
import random

import numpy as np
import torch

from raptor_t_b200 import capi, compiled, metadata, ops
from raptor_t_b200.engine import Encoder
from raptor_t_b200.modeling_bert import BertModelNoPooler

BLOCK = 64
VOCAB, TYPE_VOCAB = 50358, 2
FORBIDDEN = 12 * BLOCK  # 768 tokens: the pattern has no random table of that length, every entry point refuses it

MODELS = {
    "base": dict(hidden=768, heads=12, ffn=3072, layers=12, max_pos=4096, pattern="bigbird"),
    "band": dict(hidden=768, heads=12, ffn=3072, layers=12, max_pos=4096, pattern="band"),
    "large": dict(hidden=1024, heads=16, ffn=4096, layers=24, max_pos=8192, pattern="bigbird"),
}

_TORCH = {"f16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # one short query, answered at once: the smallest call, all latency
        dict(name="encoder_one_query", kind="encoder", model="base", dtype="f16", sequences=1, shortest=128,
             longest=128, spread="uniform", lengths=1),
        # one whole document at the model's maximum length
        dict(name="encoder_one_document", kind="encoder", model="base", dtype="f16", sequences=1, shortest=4096,
             longest=4096, spread="uniform", lengths=2),
        # a batch of paragraphs: short enough for full attention, ragged, bf16
        dict(name="encoder_paragraphs", kind="encoder", model="base", dtype="bf16", sequences=11, shortest=64,
             longest=704, spread="uniform", lengths=3),
        # the benchmark's batch of long documents
        dict(name="encoder_documents", kind="encoder", model="base", dtype="f16", sequences=8, shortest=1024,
             longest=4096, spread="uniform", lengths=4),
        # the sliding-window model's batch
        dict(name="encoder_band", kind="encoder", model="band", dtype="bf16", sequences=16, shortest=512, longest=4096,
             spread="uniform", lengths=5),
        # a GPU's share of the large model's log-normal batch: the largest call
        dict(name="encoder_large", kind="encoder", model="large", dtype="bf16", sequences=32, shortest=512,
             longest=8192, spread="lognormal", lengths=6),
        # the benchmark's batch from and to host memory
        dict(name="host_documents", kind="host", model="base", dtype="f16", sequences=8, shortest=1024, longest=4096,
             spread="uniform", lengths=7),
        # a small batch through the operator classes that replace the reference's module
        dict(name="operators_documents", kind="operators", model="base", dtype="f16", sequences=4, shortest=512,
             longest=4096, spread="uniform", lengths=8),
        # the attention kernel on a batch, and on one sequence that is longer than any batch's share of the chip
        dict(name="attention_batch", kind="attention", model="base", dtype="bf16", sequences=8, shortest=4096,
             longest=4096, spread="uniform", lengths=9),
        dict(name="attention_long", kind="attention", model="base", dtype="bf16", sequences=1, shortest=16384,
             longest=16384, spread="uniform", lengths=10),
        # a projection of a packed batch whose row count fits no tile
        dict(name="projection_ragged", kind="projection", dtype="bf16", rows=5003, columns=3072, depth=768, gelu=True),
        # the row-wise epilogue kernel at the benchmark's size
        dict(name="layernorm_rows", kind="layernorm", dtype="bf16", rows=32768, columns=768),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges, without a name."""
    kind = rng.choice(["encoder", "encoder", "encoder", "host", "operators", "attention", "projection", "layernorm"])
    dtype = rng.choice(["f16", "bf16"])
    if kind == "projection":
        columns, depth = rng.choice([(2304, 768), (768, 768), (3072, 768), (768, 3072), (4096, 1024), (1024, 4096)])
        return dict(kind=kind, dtype=dtype, rows=_log_int(rng, 64, 40000), columns=columns, depth=depth,
                    gelu=columns > depth)
    if kind == "layernorm":
        return dict(kind=kind, dtype=dtype, rows=_log_int(rng, 64, 65536), columns=rng.choice([768, 1024]))
    model = rng.choice(["base", "base", "band", "large"]) if kind == "encoder" else "base"
    top = 16384 if kind == "attention" else MODELS[model]["max_pos"]
    tokens = _log_int(rng, 128, {"encoder": 48000, "host": 24000, "operators": 24000, "attention": 65536}[kind])
    longest = min(top, max(BLOCK, _log_int(rng, 64, min(top, tokens)) // BLOCK * BLOCK))
    shortest = max(BLOCK, int(longest * rng.uniform(0.1, 1.0)) // BLOCK * BLOCK)
    if kind == "operators":  # the partition plan that these classes take needs four blocks of a sequence
        shortest, longest = max(4 * BLOCK, shortest), max(4 * BLOCK, longest)
    if shortest == longest == FORBIDDEN:
        shortest = longest = FORBIDDEN + BLOCK
    sequences = max(1, min(64, 2 * tokens // (shortest + longest)))
    return dict(kind=kind, model=model, dtype=dtype, sequences=sequences, shortest=shortest, longest=longest,
                spread="uniform", lengths=rng.randrange(1, 1 << 20))


def _lengths(case):
    """Sequence lengths of a case's batch (tokens), a function of the case alone."""
    rng = random.Random(case["lengths"])
    lo, hi = case["shortest"] // BLOCK, case["longest"] // BLOCK
    out = []
    while len(out) < case["sequences"]:
        if case["spread"] == "lognormal":
            n = min(max(math.ceil(rng.lognormvariate(math.log(2048), 0.6) / BLOCK), lo), hi)
        else:
            n = rng.randint(lo, hi)
        if n * BLOCK != FORBIDDEN:
            out.append(n * BLOCK)
    return out


def _config(case, max_pos=None, layers=None):
    m = MODELS[case["model"]]
    return capi.make_config(hidden=m["hidden"], heads=m["heads"], ffn=m["ffn"], layers=layers or m["layers"],
                            max_pos=max_pos or m["max_pos"], vocab=VOCAB, type_vocab=TYPE_VOCAB, pattern=m["pattern"],
                            dtype=case["dtype"])


def _weights(m, gen):
    """Parameters as in raptor_t_b200.weights (N(0, 0.02), perturbed biases and LayerNorms), drawn on the GPU."""
    H, F = m["hidden"], m["ffn"]

    def normal(*shape, std=0.02, mean=0.0):
        return torch.randn(*shape, device="cuda", generator=gen) * std + mean

    P = {"embeddings.word_embeddings.weight": normal(VOCAB, H),
         "embeddings.position_embeddings.weight": normal(m["max_pos"], H),
         "embeddings.token_type_embeddings.weight": normal(TYPE_VOCAB, H),
         "embeddings.LayerNorm.weight": normal(H, std=0.1, mean=1.0), "embeddings.LayerNorm.bias": normal(H, std=0.1)}
    for i in range(m["layers"]):
        pre = f"encoder.layer.{i}."
        for name, n_out, n_in in (("attention.self.query", H, H), ("attention.self.key", H, H),
                                  ("attention.self.value", H, H), ("attention.output.dense", H, H),
                                  ("intermediate.dense", F, H), ("output.dense", H, F)):
            P[pre + name + ".weight"] = normal(n_out, n_in)
            P[pre + name + ".bias"] = normal(n_out)
        for name in ("attention.output.LayerNorm", "output.LayerNorm"):
            P[pre + name + ".weight"] = normal(H, std=0.1, mean=1.0)
            P[pre + name + ".bias"] = normal(H, std=0.1)
    return P


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _TORCH[case["dtype"]]
    kind = case["kind"]
    if kind == "layernorm":
        rows, cols = case["rows"], case["columns"]
        x, res = (torch.randn(rows, cols, device="cuda", generator=gen).to(dt) for _ in range(2))
        bias, beta = ((torch.randn(cols, device="cuda", generator=gen) * 0.1).to(dt) for _ in range(2))
        gamma = (1.0 + 0.1 * torch.randn(cols, device="cuda", generator=gen)).to(dt)
        return dict(kind=kind, args=(x, bias, res, gamma, beta, 1e-12), out=torch.empty_like(x))
    if kind == "projection":
        rows, n, k = case["rows"], case["columns"], case["depth"]
        a = torch.randn(rows, k, device="cuda", generator=gen).to(dt)
        w = (torch.randn(n, k, device="cuda", generator=gen) / math.sqrt(k)).to(dt)
        bias = torch.randn(n, device="cuda", generator=gen).to(dt)
        return dict(kind=kind, args=(a, w, bias, capi.RT_EPI_BIAS_GELU if case["gelu"] else capi.RT_EPI_BIAS),
                    out=torch.empty(rows, n, device="cuda", dtype=dt))
    m, lens = MODELS[case["model"]], _lengths(case)
    T = sum(lens)
    if kind == "attention":
        cfg = _config(case, max_pos=max(m["max_pos"], max(lens)), layers=1)
        kv_ptr, kv_idx = metadata.build_block_csr(cfg, 0, lens)
        plan = ops.AttentionPlan(cfg, lens, kv_ptr, kv_idx)
        q, k, v = (torch.randn(T, m["hidden"], device="cuda", generator=gen).to(dt) for _ in range(3))
        return dict(kind=kind, args=(q, k, v, plan, 0.125), out=torch.empty_like(q))
    ids = torch.randint(5, VOCAB, (T,), device="cuda", generator=gen, dtype=torch.int32)
    P = _weights(m, gen)
    if kind == "operators":
        raptor_t = compiled.load()
        model = BertModelNoPooler.from_weights(P, m["hidden"], m["heads"], m["ffn"], m["layers"], dt, True,
                                               max_pos=m["max_pos"], pattern=m["pattern"], backend=raptor_t)
        prefix, total, part_index, part = metadata.generate_data_metainfo(lens, BLOCK, 160, m["heads"])
        pos = torch.cat([torch.arange(n, dtype=torch.int32, device="cuda") for n in lens])
        return dict(kind=kind, model=model, meta=raptor_t.MetaData(), ids=ids, pos=pos, tokens=T, prefix=prefix,
                    total=total, prefix_dev=torch.tensor(prefix, dtype=torch.int32, device="cuda"),
                    part_index=torch.from_numpy(part_index).cuda(), part=torch.from_numpy(part).cuda())
    enc = Encoder(_config(case)).load_weights(P)
    state = dict(kind=kind, encoder=enc, lens=np.asarray(lens, dtype=np.int32))
    if kind == "host":
        state["ids"] = ids.cpu().pin_memory()
        state["out"] = torch.empty(T, m["hidden"], dtype=dt).pin_memory()
    else:
        state["ids"] = ids
        state["out"] = torch.empty(T, m["hidden"], dtype=dt, device="cuda")
    return state


def run(state):
    kind = state["kind"]
    if kind == "encoder":
        return state["encoder"].prepare(state["lens"]).forward_ids(state["ids"], out=state["out"])
    if kind == "host":
        return state["encoder"].forward_host(state["lens"], state["ids"], state["out"])
    if kind == "operators":
        state["meta"].update_meta_data(state["tokens"], state["prefix"][-1] + 1, state["total"], state["prefix"])
        hidden, _ = state["model"](state["ids"], state["tokens"], 160, state["prefix"], state["prefix_dev"],
                                   state["part_index"], state["part"], position_ids=state["pos"], test_info={})
        return hidden
    if kind == "attention":
        return ops.sparse_attention(*state["args"], out=state["out"])
    if kind == "projection":
        return ops.gemm(*state["args"], out=state["out"])
    return ops.bias_residual_layernorm(*state["args"], out=state["out"])


def work(case):
    """Bytes: inputs (weights once, the embedding rows that the ids name) and outputs in 16 bits.  FLOPs: projections
    of the packed tokens and 4 * 64 * 64 * 64 per listed (query block, key block) pair and head."""
    kind = case["kind"]
    if kind == "layernorm":
        return dict(bytes=2 * (3 * case["rows"] * case["columns"] + 3 * case["columns"]),
                    flops=8 * case["rows"] * case["columns"])
    if kind == "projection":
        rows, n, k = case["rows"], case["columns"], case["depth"]
        return dict(bytes=2 * (rows * k + n * k + n + rows * n), flops=2 * rows * n * k)
    m, lens = MODELS[case["model"]], _lengths(case)
    T, H, F = sum(lens), m["hidden"], m["ffn"]
    visits = 0
    for n in lens:
        L = n // BLOCK
        if m["pattern"] == "band":
            visits += L + sum(min(L - 1, i + 4) - max(0, i - 4) + 1 + (i > 4) for i in range(1, L))
        else:
            visits += L * L if L <= 11 else 10 * L - 18
    pairs = m["heads"] * visits * 4 * BLOCK ** 3
    if kind == "attention":
        return dict(bytes=2 * 4 * T * H, flops=pairs)
    per_layer = 4 * H * H + 2 * H * F
    return dict(bytes=2 * m["layers"] * per_layer + T * (4 + 4 * H) + 4 * H * max(lens) + 2 * T * H,
                flops=m["layers"] * (2 * T * per_layer + pairs))


def tolerance(case):
    """About four times the distance (relative 2-norm) between this path and the same path in 64-bit arithmetic on the
    same 16-bit weights and inputs: encoder 0.93e-3 / 7.5e-3 (f16 / bf16), attention 2.9e-4 / 2.3e-3, projection and
    LayerNorm 2.1e-4 / 1.7e-3, the rounding of the result."""
    half = case["dtype"] == "f16"
    if case["kind"] in ("layernorm", "projection"):
        return dict(rel=8e-4 if half else 7e-3)
    if case["kind"] == "attention":
        return dict(rel=1.2e-3 if half else 1e-2)
    return dict(rel=4e-3 if half else 3.2e-2)
