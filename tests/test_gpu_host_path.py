"""The native host path (the host extension) against the Python layers (``B200Q_HOST=0``): the same entry points in the
same order, so every result has to be the same bits - linears on both sides of the GEMM rule, MoE layers with and
without pointer tables and token images, a stack, a Llama prompt and its decode steps."""

import sys

import numpy as np
import pytest

from mylocal_llm_b200 import (DevicePackedGGUFWeight, PackedMoELayer, _lib, packed_to_device, quantized_linear, synthetic_bank)
from mylocal_llm_b200.llama_model import ExternalLlamaConfig, ExternalLlamaModel
from mylocal_llm_b200.moe_stack import PackedMoEStack
from mylocal_llm_b200.quantize import random_packed
from mylocal_llm_b200.quantized_linear import dequantize_device, retile_weight

pytestmark = pytest.mark.gpu


def both(monkeypatch, run):
    """(native path, Python layers); the native path must be there."""
    assert _lib.host() is not None
    native = run()
    monkeypatch.setenv("B200Q_HOST", "0")
    assert _lib.host() is None
    python = run()
    monkeypatch.delenv("B200Q_HOST")
    return native, python


@pytest.mark.parametrize("m", [1, 8, 9, 33])
@pytest.mark.parametrize("fmt,dtype,tiled", [("Q4_K", "bfloat16", True), ("Q6_K", "bfloat16", False), ("Q8_0", "float32", True)])
def test_linear(cuda, monkeypatch, fmt, dtype, tiled, m):
    torch = cuda
    w = packed_to_device(random_packed(fmt, (80, 512), seed=m, d=0.01, dmin=0.005))
    w = retile_weight(w) if tiled else w
    x = torch.randn((1, m, 512), device="cuda").to(getattr(torch, dtype))
    for kwargs in ({}, {"out_dtype": torch.float32}, {"allow_gemm": False}):
        a, b = both(monkeypatch, lambda: quantized_linear(x, w, **kwargs))
        assert a.shape == b.shape == (1, m, 80) and a.dtype == b.dtype and torch.equal(a, b)


def test_the_gemm_rule_is_the_one_of_the_python_layers(cuda, monkeypatch):
    torch = cuda
    w = packed_to_device(random_packed("Q8_0", (128, 512), seed=1, d=0.01))
    x = torch.randn((12, 512), device="cuda").bfloat16()
    gemv, gemm = quantized_linear(x, w, allow_gemm=False), quantized_linear(x, w)
    assert not torch.equal(gemv, gemm)                          # (BF16 weights on the tensor cores)
    for yes, no in ((1, 0), (np.True_, np.False_)):
        assert torch.equal(quantized_linear(x, w, allow_gemm=yes), gemm) and torch.equal(quantized_linear(x, w, allow_gemm=no), gemv)
    model, ids = small_llama(), torch.randint(0, 512, (12, 4), device="cuda")
    step = lambda: model.prefill(ids, model.create_generation_state(12, 32))
    before = step()
    for table in ({"Q8_0": 13}, {}):
        for module in ("quantized_linear", "llama_model"):
            monkeypatch.setattr(sys.modules["mylocal_llm_b200." + module], "GEMM_MIN_TOKENS", table)
        a, b = both(monkeypatch, lambda: quantized_linear(x, w))
        assert torch.equal(a, gemv) and torch.equal(b, gemv)
        a, b = both(monkeypatch, step)
        assert torch.equal(a, b) and torch.equal(a, before) == bool(table)


@pytest.mark.parametrize("t", [1, 5, 40])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_moe_layer(cuda, monkeypatch, t, shared, dtype):
    torch = cuda
    types, d, f, e = ("Q4_K", "Q4_K", "Q6_K"), 512, 256, 16
    bank = synthetic_bank(e, d, f, types, seed=3)
    triple = tuple(packed_to_device(random_packed(q, s, seed=i, d=1 / 2048, dmin=1 / 4096))
                   for i, (q, s) in enumerate(zip(types, ((f, d), (f, d), (d, f))))) if shared else None
    gate = torch.randn(d, device="cuda") if shared else None
    layer = PackedMoELayer(bank, 0.05 * torch.randn((d, e), device="cuda"), 4, shared=triple, shared_gate=gate)
    x = torch.randn((1, t, d), device="cuda").to(getattr(torch, dtype))
    a, b = both(monkeypatch, lambda: layer.forward(x))
    assert a.dtype == b.dtype and torch.equal(a, b)


def test_a_layer_shows_what_is_replaced_after_its_first_call(cuda, monkeypatch):
    torch = cuda
    types, d, f, e = ("Q4_K", "Q4_K", "Q6_K"), 512, 256, 16
    bank, other = synthetic_bank(e, d, f, types, seed=3), synthetic_bank(e, d, f, types, seed=4)
    layer = PackedMoELayer(bank, 0.05 * torch.randn((d, e), device="cuda"), 4)
    x = torch.randn((1, 5, d), device="cuda")
    before = layer.forward(x)

    def check():
        nonlocal before
        a, b = both(monkeypatch, lambda: layer.forward(x))
        assert torch.equal(a, b) and not torch.equal(a, before)
        before = a

    layer.bank.down = PackedMoELayer(other, layer.router.W_router, 4).bank.down
    check()
    layer.router.b_router = torch.linspace(0, 3, e, device="cuda")
    check()
    layer.router.k = 2
    check()
    layer.executor.banks[0] = PackedMoELayer(other, layer.router.W_router, 4).bank
    check()
    routed, seen = layer.executor.forward_routed, []
    layer.executor.forward_routed = lambda *a, **kw: (seen.append(1), routed(*a, **kw))[1]
    assert torch.equal(layer.forward(x), before) and seen


@pytest.mark.parametrize("t", [2, 33])
def test_moe_stack(cuda, monkeypatch, t):
    torch = cuda
    stack = PackedMoEStack.synthetic(3, d_model=512, d_ff=256, n_experts=16, top_k=4, shared_d_ff=256, seed=5)
    x = torch.randn((t, 1, 512), device="cuda")
    kept = x.clone()
    a, b = both(monkeypatch, lambda: stack.forward(x))
    assert torch.equal(x, kept) and torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def test_a_stack_runs_its_layers_as_they_are(cuda, monkeypatch):
    """A subclass, a wrapped method, another epsilon, a residual of two dimensions: as on the Python layers."""
    torch = cuda
    stack = PackedMoEStack.synthetic(3, d_model=512, d_ff=256, n_experts=16, top_k=4, shared_d_ff=256, seed=5)
    x = torch.randn((7, 1, 512), device="cuda")
    with pytest.raises(ValueError, match="hidden must have shape"):
        stack.forward(x[:, 0])
    before = stack.forward(x)
    for norm in [*stack.norms, stack.final_norm]:
        norm.eps = 0.5
    a, b = both(monkeypatch, lambda: stack.forward(x))
    assert torch.equal(a[1], b[1]) and not torch.equal(a[1], before[1])
    seen, forward = [], stack.layers[1].forward
    stack.layers[1].forward = lambda *args: (seen.append("wrapped"), forward(*args))[1]
    assert torch.equal(stack.forward(x)[1], a[1]) and seen == ["wrapped"]

    class Doubled(PackedMoELayer):
        def forward(self, hidden, residual_norm=None):
            seen.append("subclass")
            return 2 * super().forward(hidden)

    del stack.layers[1].forward
    stack.layers[1].__class__ = Doubled
    assert not torch.equal(stack.forward(x)[1], a[1]) and seen[-1] == "subclass"


@pytest.mark.parametrize("batch", [1, 3, 17])
def test_llama_prompt_and_steps(cuda, monkeypatch, batch):
    torch = cuda
    cfg = ExternalLlamaConfig(vocab_size=512, hidden_size=512, intermediate_size=768, num_hidden_layers=3, num_attention_heads=8,
                              num_key_value_heads=2, head_dim=64, max_position_embeddings=128)
    model = ExternalLlamaModel.synthetic(cfg, seed=batch)
    ids = torch.randint(0, 512, (batch, 23), device="cuda")

    def run():
        state = model.create_generation_state(batch, 64)
        out = [model.prefill(ids[:, :20].contiguous(), state)] + [model.decode_one(ids[:, 20 + i].contiguous(), state) for i in range(3)]
        assert int(state.position) == state.length == 23
        return out + [state.k, state.v]

    for a, b in zip(*both(monkeypatch, run)):
        assert torch.equal(a, b)


def small_llama(layers=2, kv_heads=4, heads=4, seed=1):
    return ExternalLlamaModel.synthetic(ExternalLlamaConfig(
        vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=layers, num_attention_heads=heads,
        num_key_value_heads=kv_heads, head_dim=64, max_position_embeddings=64), seed=seed)


@pytest.mark.parametrize("host", ["1", "0"])
def test_caches_of_another_model_are_refused(cuda, monkeypatch, host):
    torch = cuda
    monkeypatch.setenv("B200Q_HOST", host)
    model, ids = small_llama(), torch.randint(0, 512, (2, 5), device="cuda")
    for other in (small_llama(layers=1), small_llama(kv_heads=1)):
        state = other.create_generation_state(2, 32)
        with pytest.raises((IndexError, RuntimeError)):
            model.prefill(ids, state)
        with pytest.raises((IndexError, ValueError)):
            model.decode_one(ids[:, 0].contiguous(), state)
    state = model.create_generation_state(2, 32)
    state.k = state.k.half()
    with pytest.raises(RuntimeError):
        model.prefill(ids, state)
    with pytest.raises(ValueError, match="KV cache"):
        model.decode_one(ids[:, 0].contiguous(), state)
    # more layers than the model has, or a strided cache in a prompt, stay what they were: fine
    state, plain = small_llama(layers=3).create_generation_state(2, 32), model.create_generation_state(2, 32)
    assert torch.equal(model.prefill(ids, state), model.prefill(ids, plain))
    assert torch.equal(state.k[:2], plain.k) and not state.k[2].any()
    strided = model.create_generation_state(2, 32)
    strided.k, strided.v = (torch.zeros((2, 2, 4, 32, 128), dtype=torch.bfloat16, device="cuda")[..., :64] for _ in range(2))
    model.prefill(ids, strided)
    assert torch.equal(strided.v[0], plain.v[0]) and torch.equal(strided.k[0], plain.k[0])


def test_what_is_replaced_after_the_first_call_counts(cuda, monkeypatch):
    """A norm weight, an epsilon, a matrix, a wrapped method: the native path gives what the Python layers give."""
    torch = cuda
    model, other, ids = small_llama(), small_llama(seed=2), torch.randint(0, 512, (2, 5), device="cuda")

    def step():
        state = model.create_generation_state(2, 32)
        return torch.stack([model.prefill(ids, state), model.decode_one(ids[:, 0].contiguous(), state)])

    def check(changed=True):
        nonlocal before
        native, python = both(monkeypatch, step)
        assert torch.equal(native, python) and torch.equal(native, before) != changed
        before = native

    before = step()
    check(changed=False)
    gamma = torch.linspace(0.5, 1.5, 256, device="cuda").bfloat16()
    model.layers[1]["norm2"].set_weights(gamma)
    check()
    model.final_norm.eps = 0.1
    check()
    model.layers[0]["down"] = other.layers[0]["down"]
    check()
    model.lm_head = other.lm_head
    check()
    model.layers[0]["norm1"].set_weights(gamma.float())          # another type: the Python layers take it
    check()
    model.layers[0]["norm1"].set_weights(gamma)
    check()
    linear, seen = model._linear, []
    model._linear = lambda *a: (seen.append(1), linear(*a))[1]
    check(changed=False)
    assert seen


@pytest.mark.parametrize("bad", [512, -1, 2 ** 40])
def test_a_token_outside_the_vocabulary_shows_in_its_sequence(cuda, bad):
    """(By the kernel's own bounds check; the native path only.)"""
    torch = cuda
    model, ids = small_llama(), torch.randint(0, 512, (3, 6), device="cuda")
    assert model._native(ids, model.create_generation_state(3, 32)) is not None
    good, state = model.create_generation_state(3, 32), model.create_generation_state(3, 32)
    want = model.prefill(ids, good)
    ids[1, 2] = bad
    logits = model.prefill(ids, state)
    assert torch.isnan(logits[1]).all() and torch.equal(logits[0], want[0]) and torch.equal(logits[2], want[2])
    step = torch.tensor([5, 6, bad], device="cuda")
    logits = model.decode_one(step, good)
    assert torch.isnan(logits[2]).all() and torch.isfinite(logits[:2]).all()
    assert _lib.device_status() == 302
    _lib.clear_device_status()


@pytest.mark.parametrize("fmt", ["Q8_0", "Q4_K", "Q6_K"])
def test_embed_rows_is_the_gather_of_dequantised_rows(cuda, fmt):
    torch = cuda
    import ctypes
    w = packed_to_device(random_packed(fmt, (37, 512), seed=1, d=0.01, dmin=0.005))
    ids = torch.tensor([36, 0, 5, 5, 17], device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    out = torch.full((6, 512), float("nan"), device="cuda")
    _lib.call("b200q_embed_rows", ptr(w.data), _lib.FORMAT_ID[fmt], 37, 512, ptr(ids), 5, ptr(out), _lib.current_stream())
    assert torch.equal(out[:5], dequantize_device(w.data, 37, 512, fmt)[ids]) and torch.isnan(out[5]).all()
    assert _lib.device_status() == 0
    bad = torch.tensor([37, 3], device="cuda")
    _lib.call("b200q_embed_rows", ptr(w.data), _lib.FORMAT_ID[fmt], 37, 512, ptr(bad), 2, ptr(out), _lib.current_stream())
    assert _lib.device_status() == 302 and (out[0] == 0).all()          # refused by the kernel's own bounds check
    _lib.clear_device_status()


def test_calls_stay_visible_when_they_are_intercepted(cuda):
    torch = cuda
    w = packed_to_device(random_packed("Q8_0", (64, 256), seed=2, d=0.01))
    real, calls = _lib.call, []
    _lib.call = lambda name, *a: (calls.append(name), real(name, *a))[1]
    try:
        quantized_linear(torch.zeros((1, 256), device="cuda"), w)
    finally:
        _lib.call = real
    assert calls == ["b200q_gemv"]


def test_errors_are_those_of_the_python_layer(cuda):
    torch = cuda
    w = DevicePackedGGUFWeight(torch.zeros(64 * 34, dtype=torch.uint8, device="cuda"), (64, 32), "Q8_0")
    with pytest.raises(ValueError, match="K does not match"):
        quantized_linear(torch.zeros((1, 64), device="cuda"), w)
    with pytest.raises(ValueError, match="contiguous"):
        quantized_linear(torch.zeros((32, 2), device="cuda").t(), w)
    with pytest.raises(TypeError):
        quantized_linear(np.zeros((1, 32), np.float32), w)
    with pytest.raises(TypeError, match="FP16, BF16, or FP32"):
        quantized_linear(torch.zeros((1, 32), dtype=torch.float64, device="cuda"), w)


@pytest.mark.parametrize("what", ["linear", "layer", "stack", "prefill", "decode"])
def test_other_threads_run_while_a_launch_waits(cuda, what):
    """A launch into a full queue waits for the GPU; the interpreter's lock is free meanwhile, as it is in a ctypes call."""
    torch = cuda
    import threading
    import time
    if what == "linear":
        w = packed_to_device(random_packed("Q8_0", (64, 256), seed=2, d=0.01))
        x = torch.zeros((1, 256), device="cuda")
        run, calls = lambda: quantized_linear(x, w), 3000
    elif what in ("layer", "stack"):
        stack = PackedMoEStack.synthetic(2, d_model=512, d_ff=256, n_experts=16, top_k=4, shared_d_ff=256, seed=5)
        x = torch.randn((3, 1, 512), device="cuda")
        run, calls = (lambda: stack.forward(x)) if what == "stack" else (lambda: stack.layers[0].forward(x)), 400
    else:
        model, ids = small_llama(), torch.zeros((2, 4), dtype=torch.int64, device="cuda")
        state = model.create_generation_state(2, 64)
        run, calls = (lambda: model.prefill(ids, state)) if what == "prefill" else (
            lambda: (setattr(state, "length", 0), state.position.zero_(), model.decode_one(ids[:, 0].contiguous(), state))), 150
    run()
    torch.cuda.synchronize()
    gaps, done = [0.0], threading.Event()

    def watch():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    thread = threading.Thread(target=watch)
    thread.start()
    torch.cuda._sleep(1_500_000_000)                    # most of a second
    t0 = time.perf_counter()
    for _ in range(calls):
        run()
    waited = time.perf_counter() - t0
    done.set()
    thread.join()
    torch.cuda.synchronize()
    assert waited > 0.4, "the queue did not fill"
    assert max(gaps) < waited / 2, (max(gaps), waited)          # (one call waits nearly all of it)
