"""What this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values; ``listed()`` names the standing ones, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call (packed weights, inputs, caches, a captured graph),
``run(state)`` is one pass through the public entry points and ``work(case)`` the bytes and operations that pass cannot
do without. Four kinds of use:

``linear``   ``quantized_linear`` on packed GGUF matrices: one matrix or the matrices of a few layers in a row. Decode
             calls (a few tokens) read the device tile layouts where one exists (``tiled``), prefill calls the GGUF bytes.
``moe``      one ``PackedMoELayer`` (router, routed experts, shared expert) on a batch of hidden states.
``stack``    one step of a ``PackedMoEStack``: norms, MoE layers and the FP32 residual stream.
``prefill``  ``ExternalLlamaModel.prefill``: the prompt of one or several sequences.
``decode``   ``ExternalLlamaModel.decode_one``, a few steps in a row from a filled cache, either called directly or
             captured once in a CUDA graph and replayed.
"""

import math

import torch

from mylocal_llm_b200 import DevicePackedGGUFWeight, PackedExpertBank, PackedMoELayer, RMSNormInference, quantized_linear
from mylocal_llm_b200.llama_model import ExternalLlamaConfig, ExternalLlamaModel
from mylocal_llm_b200.moe_stack import PackedMoEStack
from mylocal_llm_b200.quantized_linear import retile_weight

BLOCK = {"Q8_0": (32, 34), "Q4_K": (256, 144), "Q5_K": (256, 176), "Q6_K": (256, 210)}
EXPERT_TYPES = ("Q4_K", "Q4_K", "Q6_K")          # gate, up, down
ESIZE = {"float32": 4, "float16": 2, "bfloat16": 2}
NEW_TOKENS = 128                                 # cache positions kept free behind a prompt
DECODE_STEPS = 4                                 # decode steps of one pass


# ------------------------------------------------------------------------------------------------ cases
def _linear(fmt, n, k, m, dtype="bfloat16", tiled=False, layers=1):
    return {"kind": "linear", "fmt": fmt, "n": n, "k": k, "m": m, "dtype": dtype, "tiled": tiled, "layers": layers}


def _moe(tokens, layers=1, kind="moe", experts=512, top_k=10, d_model=2048, d_ff=512, dtype="bfloat16"):
    return {"kind": kind, "tokens": tokens, "layers": layers, "experts": experts, "top_k": top_k, "d_model": d_model,
            "d_ff": d_ff, "dtype": dtype}


def _llama(kind, batch, context, layers=24, kv_heads=32, graph=False):
    return {"kind": kind, "batch": batch, "context": context, "layers": layers, "kv_heads": kv_heads, "graph": graph}


def listed():
    cases = {
        # a single projection for a single token, FP32 activations: the smallest call there is
        "linear_q8_0_4096x4096_m1": _linear("Q8_0", 4096, 4096, 1, "float32", tiled=True),
        # the same projection of eight layers for a decode batch of eight sequences
        "linear_q4_k_8192x2048_m8": _linear("Q4_K", 8192, 2048, 8, tiled=True, layers=8),
        # a short ragged batch of tokens on a matrix whose rows fill no tile
        "linear_q6_k_5003x2816_m77": _linear("Q6_K", 5003, 2816, 77),
        # a prompt's worth of tokens through one projection
        "linear_q5_k_8192x2048_m512": _linear("Q5_K", 8192, 2048, 512),
        # one MoE layer: a small decode batch, and a large batch or a short prompt
        "moe_layer_t16": _moe(16),
        "moe_layer_t256": _moe(256),
        # a decode step through a stack of MoE layers: one sequence, and a serving batch
        "moe_stack_t1": _moe(1, 8, "stack"),
        "moe_stack_t64": _moe(64, 8, "stack"),
        # a 1.7B decoder: one prompt (time to first token) and a batch of prompts
        "prefill_b1_t512": _llama("prefill", 1, 512),
        "prefill_b16_t512": _llama("prefill", 16, 512),
        # decode steps of that model: one sequence replayed from a graph, a batch called directly
        "decode_b1_c512": _llama("decode", 1, 512, graph=True),
        "decode_b16_c512": _llama("decode", 16, 512),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "moe", "moe", "stack", "stack", "prefill", "prefill", "decode", "decode"))
    if kind == "linear":
        fmt = rng.choice(tuple(BLOCK))
        unit = BLOCK[fmt][0] if rng.random() < 0.3 else 256
        k = unit * _log_int(rng, 256 // unit, 8192 // unit)
        n = _log_int(rng, 256, 49152)
        if rng.random() < 0.7:
            n = max(256, n // 64 * 64)
        if rng.random() < 0.5:                                     # decode: a few tokens, the decode layout
            return _linear(fmt, n, k, rng.randint(1, 8), rng.choice(("bfloat16", "bfloat16", "float16", "float32")), True,
                           rng.choice((1, 1, 4, 8)))
        return _linear(fmt, n, k, _log_int(rng, 9, 2048))          # batched decode or prefill
    if kind in ("moe", "stack"):
        tokens = rng.choice((1, _log_int(rng, 2, 64), _log_int(rng, 2, 64))) if kind == "stack" else _log_int(rng, 1, 512)
        return _moe(tokens, rng.randint(2, 8) if kind == "stack" else 1, kind, rng.choice((128, 256, 512)),
                    rng.choice((4, 8, 10)), rng.choice((1024, 2048)), rng.choice((256, 512, 768)),
                    "bfloat16" if kind == "stack" or rng.random() < 0.7 else "float32")
    layers, kv_heads = rng.randint(4, 24), rng.choice((32, 32, 8))
    if kind == "prefill":
        context = _log_int(rng, 16, 1900)
        batch = rng.choice((1, 1, _log_int(rng, 2, 16)))
        return _llama(kind, max(1, min(batch, 8192 // context)), context, min(layers, 12) if context > 1000 else layers,
                      kv_heads)
    return _llama(kind, rng.choice((1, 1, _log_int(rng, 2, 16))), _log_int(rng, 16, 1900), layers, kv_heads,
                  rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------ inputs
def _packed(fmt, rows, k, gen, sd=0.02):
    """Packed bytes of a ``[rows, k]`` matrix on the GPU: uniform codes and sub-block scales, block scales that spread
    by a factor of 1.7 and make the weights zero-mean with a standard deviation of about ``sd``."""
    qk, qb = BLOCK[fmt]
    blocks = rows * k // qk
    raw = torch.randint(0, 256, (blocks, qb), dtype=torch.uint8, device="cuda", generator=gen)
    d = 0.75 + 0.5 * torch.rand(blocks, 1, device="cuda", generator=gen)
    half = lambda v: v.to(torch.float16).view(torch.uint8)
    if fmt == "Q8_0":
        raw[:, 0:2] = half(d * (sd / 74.0))
    elif fmt == "Q6_K":
        raw[:, 208:210] = half(d * (sd / 1366.0))
    else:
        steps = 15 if fmt == "Q4_K" else 31
        raw[:, 0:2] = half(d * (sd / (14.2 * (steps + 1))))
        raw[:, 2:4] = half(d * (sd / (14.2 * (steps + 1)) * steps / 2))
    return raw.reshape(-1)


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _moe_layer(case, gen, index):
    e, d, f = case["experts"], case["d_model"], case["d_ff"]
    shapes = ((f, d), (f, d), (d, f))
    bank = PackedExpertBank(*(_packed(fmt, e * n, k, gen) for fmt, (n, k) in zip(EXPERT_TYPES, shapes)), *EXPERT_TYPES, e, d, f)
    shared = tuple(DevicePackedGGUFWeight(_packed(fmt, n, k, gen), (n, k), fmt) for fmt, (n, k) in zip(EXPERT_TYPES, shapes))
    router = 0.02 * torch.randn(d, e, device="cuda", generator=gen)
    return PackedMoELayer(bank, router, case["top_k"], shared=shared, layer_id=index)


def _llama_config(case):
    return ExternalLlamaConfig(vocab_size=49152, hidden_size=2048, intermediate_size=8192, num_hidden_layers=case["layers"],
                               num_attention_heads=32, num_key_value_heads=case["kv_heads"], head_dim=64,
                               max_position_embeddings=2048, rope_theta=10000.0, rms_norm_eps=1e-5)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "linear":
        n, k, dtype = case["n"], case["k"], getattr(torch, case["dtype"])
        weights = [DevicePackedGGUFWeight(_packed(case["fmt"], n, k, gen), (n, k), case["fmt"]) for _ in range(case["layers"])]
        if case["tiled"]:
            weights = [retile_weight(w, force=dtype != torch.float32) for w in weights]
        state.update(weights=weights, x=torch.randn(case["m"], k, device="cuda", generator=gen).to(dtype))
        return state
    if kind in ("moe", "stack"):
        d, dtype = case["d_model"], getattr(torch, case["dtype"])
        layers = [_moe_layer(case, gen, i) for i in range(case["layers"])]
        x = torch.randn(1, case["tokens"], d, device="cuda", generator=gen)
        if kind == "moe":
            state.update(layer=layers[0], x=x.to(dtype))
            return state
        norms = [RMSNormInference(d, eps=1e-5) for _ in range(len(layers) + 1)]
        for norm in norms:
            norm.set_weights((1 + 0.1 * torch.randn(d, device="cuda", generator=gen)).to(dtype))
        state.update(stack=PackedMoEStack(layers, norms[:-1], norms[-1]), x=x.reshape(case["tokens"], 1, d))
        return state
    model = ExternalLlamaModel.synthetic(_llama_config(case), seed=seed % 1000003)
    b, context = case["batch"], case["context"]
    cache = model.create_generation_state(b, context + NEW_TOKENS)
    state.update(model=model, cache=cache, context=context)
    if kind == "prefill":
        state["ids"] = torch.randint(0, 49152, (b, context), device="cuda", generator=gen)
        return state
    for part in (cache.k, cache.v):              # the rows that a prompt has left
        for layer in part:
            layer[:, :, :context].normal_(0.0, 1.0, generator=gen)
    state["ids"] = torch.randint(0, 49152, (DECODE_STEPS, b), device="cuda", generator=gen)
    if case["graph"]:
        # the usual capture: warm up on a side stream, record one step, replay it for every token
        token, stream = state["ids"][0].clone(), torch.cuda.Stream()
        cache.position.fill_(context)
        cache.length = context
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            model.decode_one(token, cache)
        torch.cuda.current_stream().wait_stream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = model.decode_one(token, cache)
        state.update(token=token, graph=graph, graph_logits=logits,
                     logits=torch.empty((DECODE_STEPS,) + tuple(logits.shape), device="cuda"))
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return [quantized_linear(state["x"], w) for w in state["weights"]]
    if kind == "moe":
        return state["layer"].forward(state["x"])
    if kind == "stack":
        return state["stack"].forward(state["x"])
    model, cache = state["model"], state["cache"]
    if kind == "prefill":
        logits = model.prefill(state["ids"], cache)
        return {"logits": logits, "k": cache.k, "v": cache.v}
    cache.position.fill_(state["context"])       # back to the end of the prompt
    cache.length = state["context"]
    if "graph" in state:
        logits = state["logits"]
        for i in range(DECODE_STEPS):
            state["token"].copy_(state["ids"][i])
            state["graph"].replay()
            logits[i].copy_(state["graph_logits"])
    else:
        logits = [model.decode_one(state["ids"][i], cache) for i in range(DECODE_STEPS)]
    return {"logits": logits, "k": cache.k, "v": cache.v}


def _bytes(fmt, n, k):
    qk, qb = BLOCK[fmt]
    return n * k // qk * qb


def work(case):
    kind = case["kind"]
    if kind == "linear":
        n, k, m, es = case["n"], case["k"], case["m"], ESIZE[case["dtype"]]
        return {"bytes": case["layers"] * (_bytes(case["fmt"], n, k) + m * n * es) + m * k * es,
                "flops": 2.0 * m * n * k * case["layers"]}
    if kind in ("moe", "stack"):
        t, e, k, d, f = case["tokens"], case["experts"], case["top_k"], case["d_model"], case["d_ff"]
        expert = sum(_bytes(fmt, *s) for fmt, s in zip(EXPERT_TYPES, ((f, d), (f, d), (d, f))))
        active = e * (1.0 - (1.0 - k / e) ** t) + 1                # experts that some token has chosen, and the shared one
        rows = 2 * t * d * (4 if kind == "stack" else ESIZE[case["dtype"]])
        return {"bytes": case["layers"] * (active * expert + 4.0 * d * e) + rows,
                "flops": case["layers"] * (2.0 * t * (k + 1) * 3 * d * f + 2.0 * t * d * e)}
    d, f, v, layers = 2048, 8192, 49152, case["layers"]
    b, c, kv = case["batch"], case["context"], case["kv_heads"] * 64
    linears = 2 * d * d + 2 * kv * d + 3 * f * d
    packed = layers * _bytes("Q8_0", linears // d, d) + _bytes("Q8_0", v, d)
    if kind == "prefill":
        return {"bytes": packed + layers * 2 * b * c * kv * 2 + b * c * 2210 + b * v * 4,
                "flops": 2.0 * b * c * linears * layers + layers * 2.0 * b * c * (c + 1) * d + 2.0 * b * v * d}
    return {"bytes": DECODE_STEPS * (packed + layers * 2 * b * (c + 2) * kv * 2 + b * v * 4),
            "flops": DECODE_STEPS * b * (2.0 * linears * layers + 2.0 * v * d + layers * 4.0 * (c + 2) * d)}


def tolerance(case):
    dtype = case.get("dtype", "bfloat16")
    if case["kind"] == "linear":
        # FP32: 32-bit sums. 16-bit: the output's rounding, and BF16 weights where the tensor cores take many tokens.
        return {"rel": {"float32": 2e-5, "float16": 2e-3, "bfloat16": 1e-2}[dtype]}
    if case["kind"] == "moe" and dtype == "float32":
        return {"rel": 1e-4}                     # three chained products and an exponential in FP32
    return {"rel": 1e-2, "max": 0.5}             # BF16 activations between the layers
