"""Grouped projections over images (``grouped_stream.cu``) against the block-structured kernels (``B200Q_TOKEN_IMAGES=0``):
the same sums, so equal bits - segments of one to eight tokens, experts of several segments, experts without any, one to
many row groups per segment (fewer than a CTA has teams included), one to nine super-blocks per row, every team size."""

import pytest

from mylocal_llm_b200 import moe_ops
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


@pytest.mark.parametrize("tokens,e,k", [(17, 7, 2), (40, 24, 4), (33, 120, 3), (64, 96, 6), (256, 40, 8)])
@pytest.mark.parametrize("d,f", [(256, 16), (2048, 48), (768, 512), (2304, 256)])
def test_same_bits_as_the_block_kernels(cuda, monkeypatch, tokens, e, k, d, f):
    torch = cuda
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
