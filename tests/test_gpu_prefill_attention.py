"""Prompt attention (``b200q_prefill_attention``): rotated keys and plain values in the caches, and causal attention
against an FP64 reference over those caches (mini_llm/ops/attention_inference.py:255-277), at the edges of the row
and position tiles, with grouped KV heads and a cache tail of NaN that must never enter the sums.

Bound of the output: its own BF16 rounding (half a unit in the last of eight bits: at most 2^-8 of the value) plus the FP32 sums - scores of |q||k| / 8 of
about 8 * 2^-24 each, through the exponential and a weighted mean of values of order one: below 2e-5 absolute."""

import ctypes

import pytest

from mylocal_llm_b200 import _lib

pytestmark = pytest.mark.gpu


def rotate(x, cos, sin):
    half = x.shape[-1] // 2
    x0, x1 = x[..., :half], x[..., half:]
    c, s = cos[None, :, None, :], sin[None, :, None, :]
    return (x0 * c - x1 * s, x0 * s + x1 * c)


@pytest.mark.parametrize("batch,heads,kv_heads,dh", [(1, 4, 4, 64), (3, 8, 2, 64)])
@pytest.mark.parametrize("t", [2, 15, 64, 65, 129, 300, 640, 641, 1000])
def test_prompt_attention_matches_fp64(cuda, batch, heads, kv_heads, dh, t):
    torch = cuda
    horizon = t + 9
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000 * t + 10 * heads + batch)
    qkv = torch.randn((batch * t, (heads + 2 * kv_heads) * dh), device="cuda", generator=gen)
    q, k, v = qkv[:, :heads * dh], qkv[:, heads * dh:(heads + kv_heads) * dh], qkv[:, (heads + kv_heads) * dh:]
    angle = torch.arange(horizon, device="cuda")[:, None] * (10000.0 ** (-2.0 * torch.arange(dh // 2, device="cuda") / dh))
    cos, sin = torch.cos(angle), torch.sin(angle)
    kc, vc = (torch.full((batch, kv_heads, horizon, dh), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    out = torch.empty((batch * t, heads * dh), dtype=torch.bfloat16, device="cuda")
    ptr = lambda x: ctypes.c_void_p(x.data_ptr())
    _lib.call("b200q_prefill_attention", ptr(q), ptr(k), ptr(v), qkv.stride(0), qkv.stride(0), qkv.stride(0), ptr(cos),
              ptr(sin), horizon, batch, t, heads, kv_heads, dh, horizon, ptr(kc), ptr(vc), 2, float(dh ** -0.5), ptr(out), 2,
              _lib.current_stream())
    torch.cuda.synchronize()
    assert torch.isnan(kc[:, :, t:].float()).all() and torch.isnan(vc[:, :, t:].float()).all()
    cd, sd = cos[:t].double(), sin[:t].double()
    kr = torch.cat(rotate(k.double().reshape(batch, t, kv_heads, dh), cd, sd), -1).permute(0, 2, 1, 3)
    # one BF16 rounding of an FP32 rotation (two roundings of 2^-24)
    assert ((kc[:, :, :t].double() - kr).abs() <= kr.abs() * 2.0 ** -8 + 1e-6).all()
    assert torch.equal(vc[:, :, :t], v.reshape(batch, t, kv_heads, dh).permute(0, 2, 1, 3).to(torch.bfloat16))
    qr = torch.cat(rotate(q.double().reshape(batch, t, heads, dh), cd, sd), -1).permute(0, 2, 1, 3)
    group = heads // kv_heads
    keys = kc[:, :, :t].double().repeat_interleave(group, 1)
    values = vc[:, :, :t].double().repeat_interleave(group, 1)
    scores = qr @ keys.transpose(-1, -2) * dh ** -0.5
    mask = torch.ones((t, t), dtype=torch.bool, device="cuda").tril()
    ref = torch.softmax(scores.masked_fill(~mask, float("-inf")), -1) @ values
    got = out.reshape(batch, t, heads, dh).permute(0, 2, 1, 3).double()
    assert ((got - ref).abs() <= ref.abs() * 2.0 ** -8 + 2e-5).all()


def test_unsupported_forms_are_refused(cuda):
    assert _lib.load().b200q_prefill_attention_supported(8, 2, 64, 100, 1024, 2, 2) == 1
    for args in ((8, 3, 64, 100, 200, 2, 2), (8, 2, 128, 100, 200, 2, 2), (8, 2, 64, 100, 200, 1, 1), (8, 2, 64, 100, 99, 2, 2),
                 (8, 2, 64, 100, 1025, 2, 2)):
        assert _lib.load().b200q_prefill_attention_supported(*args) == 0


@pytest.mark.parametrize("t,bad", [(70, 40), (300, 0), (600, 599)])
def test_a_row_of_nan_reaches_the_rows_that_see_it(cuda, t, bad):
    """... and the other sequence keeps its bits; so does every row block that ends before it."""
    torch = cuda
    batch, heads, dh = 2, 4, 64
    angle = torch.arange(t, device="cuda")[:, None] * (10000.0 ** (-2.0 * torch.arange(dh // 2, device="cuda") / dh))
    cos, sin = torch.cos(angle), torch.sin(angle)
    qkv = torch.randn((batch * t, 3 * heads * dh), device="cuda")
    ptr = lambda x: ctypes.c_void_p(x.data_ptr())

    def run():
        kc, vc = (torch.zeros((batch, heads, t, dh), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        out = torch.empty((batch, t, heads * dh), dtype=torch.bfloat16, device="cuda")
        q, k, v = qkv.split(heads * dh, dim=1)
        _lib.call("b200q_prefill_attention", ptr(q), ptr(k), ptr(v), qkv.stride(0), qkv.stride(0), qkv.stride(0), ptr(cos),
                  ptr(sin), t, batch, t, heads, heads, dh, t, ptr(kc), ptr(vc), 2, float(dh ** -0.5), ptr(out), 2,
                  _lib.current_stream())
        return out

    clean = run()
    qkv[bad] = float("nan")
    out = run()
    assert torch.isnan(out[0, bad:]).all() and torch.equal(out[1], clean[1]) and torch.isfinite(clean).all()
    before = bad // 64 * 64                              # (row blocks of 32 or 64)
    assert torch.equal(out[0, :before], clean[0, :before])
