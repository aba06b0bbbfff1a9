"""Grouped projections over images (``grouped_stream.cu``) against the block-structured kernels (``B200Q_TOKEN_IMAGES=0``):
the same sums, so equal bits - segments of one to eight tokens, experts of several segments, experts without any, one to
many row groups per segment (fewer than a CTA has teams included), one to nine super-blocks per row, every team size."""

import pytest

from mylocal_llm_b200 import _lib, moe_ops
from mylocal_llm_b200.quantize import random_packed
from mylocal_llm_b200.quantized_linear import retile_bytes

pytestmark = pytest.mark.gpu


def bank(torch, fmt, e, n, k, seed):
    packed = random_packed(fmt, (e * n, k), seed=seed, d=1 / 2048, dmin=1 / 4096)
    data = torch.from_numpy(packed.data.reshape(-1).copy()).cuda()
    return retile_bytes(data, e * n, k, fmt), data.numel() // e


def both(monkeypatch, run):
    images = run()
    monkeypatch.setenv("B200Q_TOKEN_IMAGES", "0")
    plain = run()
    monkeypatch.delenv("B200Q_TOKEN_IMAGES")
    return images, plain


@pytest.mark.parametrize("tokens,e,k", [(17, 7, 2), (40, 24, 4), (33, 120, 3), (64, 96, 6), (256, 40, 8), (45, 120, 3), (70, 300, 3)])
@pytest.mark.parametrize("d,f", [(256, 16), (2048, 48), (768, 512), (2304, 256)])
def test_same_bits_as_the_block_kernels(cuda, monkeypatch, tokens, e, k, d, f):
    torch = cuda
    monkeypatch.setenv("B200Q_GROUPED_STREAM", "1")                     # also where the block-structured kernels are faster
    gen = torch.Generator(device="cuda")
    gen.manual_seed(tokens + d)
    scores = torch.rand((tokens, e), device="cuda", generator=gen)
    scores[:, 0] += 0.4                                                 # a crowded expert
    ids = torch.topk(scores, k).indices
    plan = moe_ops.moe_plan(ids, e)
    for fmt, dtype in (("Q4_K", "bfloat16"), ("Q5_K", "float32")):
        x = torch.randn((tokens, d), device="cuda", generator=gen).to(getattr(torch, dtype))
        (gate, stride), (up, _) = bank(torch, fmt, e, f, d, 1), bank(torch, fmt, e, f, d, 2)
        a, b = both(monkeypatch, lambda: moe_ops.moe_gate_up(x, plan, gate, up, fmt + "_TILED", fmt + "_TILED", f, d, stride, stride))
        assert torch.isfinite(a).all() and torch.equal(a, b)
    route = torch.rand((tokens, k), device="cuda", generator=gen)
    wide = (f + 255) // 256 * 256                                       # hidden width of the down projection
    hidden = torch.randn((tokens * k, wide), device="cuda", generator=gen)
    for fmt in ("Q6_K", "Q8_0"):
        down, stride = bank(torch, fmt, e, d, wide, 3)
        for flat in (False, True):
            a, b = both(monkeypatch, lambda: moe_ops.moe_down(hidden, route, plan, down, fmt + "_TILED", d, wide, stride, flat_rows=flat))
            assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("tokens,e,k,d,f,fmts,gate_up,down", [
    (2, 64, 5, 1024, 512, ("Q4_K", "Q6_K"), 0, 0),             # 11 segments at most: the block-structured kernels
    (8, 64, 5, 1024, 512, ("Q4_K", "Q6_K"), 0, 1),             # 45
    (8, 64, 5, 1024, 512, ("Q4_K", "Q8_0"), 0, 1),
    (24, 64, 5, 1024, 2048, ("Q5_K", "Q6_K"), 0, 0),           # rows of 2048 hidden values: no room for the tile rings
    (32, 64, 5, 1024, 512, ("Q4_K", "Q6_K"), 1, 1),            # 84: token images for the block-structured gate/up
    (16, 512, 11, 1024, 512, ("Q4_K", "Q6_K"), 1, 1),          # 198: both stream
])
def test_images_are_made_for_the_launches_that_read_them(cuda, tokens, e, k, d, f, fmts, gate_up, down):
    torch = cuda
    ids = torch.rand((tokens, e), device="cuda").topk(k, dim=1).indices.contiguous()
    plan = moe_ops.moe_plan(ids, e)
    x = torch.randn((tokens, d), device="cuda").bfloat16()
    (gate, stride), (up, _), (down_bank, down_stride) = (bank(torch, fmt, e, n, w, s) for fmt, n, w, s in (
        (fmts[0], f, d, 1), (fmts[0], f, d, 2), (fmts[1], d, f, 3)))
    real, calls = _lib.call, []
    _lib.call = lambda name, *a: (calls.append(name), real(name, *a))[1]
    try:
        hidden = moe_ops.moe_gate_up(x, plan, gate, up, fmts[0] + "_TILED", fmts[0] + "_TILED", f, d, stride, stride)
        moe_ops.moe_down(hidden, torch.rand((tokens, k), device="cuda"), plan, down_bank, fmts[1] + "_TILED", d, f, down_stride)
    finally:
        _lib.call = real
    assert (calls.count("b200q_moe_token_images"), calls.count("b200q_moe_hidden_images")) == (gate_up, down)


def test_infinities_and_nan_are_those_of_the_block_kernels(cuda, monkeypatch):
    """Rows with an infinity, a NaN, only zeros or the type's largest magnitude, in the images and in what is computed."""
    torch = cuda
    tokens, e, k, d, f = 64, 96, 6, 2048, 512                           # 144 segments: both launches stream
    ids = torch.rand((tokens, e), device="cuda").topk(k, dim=1).indices.contiguous()
    plan = moe_ops.moe_plan(ids, e)
    assert _lib.load().b200q_moe_gate_up_streams(_lib.FORMAT_ID["Q4_K_TILED"], f, d, 2, plan.max_segments)
    assert _lib.load().b200q_moe_down_streams(_lib.FORMAT_ID["Q6_K_TILED"], d, f, plan.max_segments)

    def odd(rows, width, dtype):
        x = torch.randn((rows, width), device="cuda").to(dtype)
        x[3, 5], x[9, 7], x[11], x[20, 1], x[33, 0] = float("inf"), float("nan"), 0, torch.finfo(dtype).max, -float("inf")
        return x

    (gate, stride), (up, _) = bank(torch, "Q4_K", e, f, d, 1), bank(torch, "Q4_K", e, f, d, 2)
    x = odd(tokens, d, torch.bfloat16)
    a, b = both(monkeypatch, lambda: moe_ops.moe_gate_up(x, plan, gate, up, "Q4_K_TILED", "Q4_K_TILED", f, d, stride, stride))
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(), b.nan_to_num()) and torch.isnan(a).any()
    down, stride = bank(torch, "Q6_K", e, d, f, 3)
    hidden, route = odd(tokens * k, f, torch.float32), torch.rand((tokens, k), device="cuda")
    a, b = both(monkeypatch, lambda: moe_ops.moe_down(hidden, route, plan, down, "Q6_K_TILED", d, f, stride))
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(), b.nan_to_num()) and torch.isnan(a).any()
    assert torch.isfinite(a[50:]).all()
