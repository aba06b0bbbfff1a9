"""Preparation of the activations of several tokens (``prepare_tokens``): a token's result must not depend on how many
tokens a launch carries, so every row of a batch equals the launch of that row alone, bit for bit - at token counts and
K on both sides of the chunk rule, with partial batches of chunks, 16-bit and FP32 inputs, rows of zeros, of the largest
and smallest magnitudes, and an activation pointer that is not aligned for vector loads."""

import pytest

from mylocal_llm_b200 import packed_to_device, quantized_linear
from mylocal_llm_b200.quantize import random_packed
from mylocal_llm_b200.quantized_linear import retile_weight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
@pytest.mark.parametrize("dtype", ["bfloat16", "float16", "float32"])
@pytest.mark.parametrize("k", [256, 1024, 2304, 4096])
def test_rows_of_a_batch_are_the_single_rows(cuda, fmt, dtype, k):
    torch = cuda
    w = retile_weight(packed_to_device(random_packed(fmt, (80, k), seed=k, d=0.01, dmin=0.005)), force=True)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(k)
    x = torch.randn((16, k), device="cuda", generator=gen)
    x[3] = 0.0
    x[5] *= 1e4
    x[6] *= 1e-6
    x[7, k // 2] = 6e4
    x = x.to(getattr(torch, dtype))
    single = torch.cat([quantized_linear(x[i:i + 1], w, allow_gemm=False) for i in range(16)])
    for m in (2, 3, 7, 8, 9, 13, 16):
        assert torch.equal(quantized_linear(x[:m], w, allow_gemm=False), single[:m])
    odd = torch.empty(8 * k + 1, dtype=x.dtype, device="cuda")[1:].view(8, k)
    odd.copy_(x[:8])
    assert torch.equal(quantized_linear(odd, w, allow_gemm=False), single[:8])


def test_a_row_of_nan_or_infinity_stays_its_own(cuda):
    torch = cuda
    for fmt in ("Q4_K", "Q8_0"):
        w = retile_weight(packed_to_device(random_packed(fmt, (64, 2048), seed=1, d=0.01, dmin=0.005)), force=True)
        x = torch.randn((8, 2048), device="cuda").to(torch.bfloat16)
        clean = quantized_linear(x, w)
        x[2, 100] = float("nan")
        x[4] = float("inf")
        y = quantized_linear(x, w)
        keep = [0, 1, 3, 5, 6, 7]
        assert torch.equal(y[keep], clean[keep]) and torch.isnan(y[2].float()).all() and not torch.isfinite(y[4].float()).any()
