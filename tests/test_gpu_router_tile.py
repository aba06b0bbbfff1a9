"""Router logits from register tiles (many tokens) against the same rows through calls of a few tokens, which take the
other kernel and the same order of sums: equal bits, at the edges of the row and token tiles and of the 128 columns of a
step, with and without a bias, and against FP64. FP64 bound: a chain of d / 32 FMAs, five adds of lanes and the bias, each
2^-24 of the sum of magnitudes at most."""

import pytest

from mylocal_llm_b200 import moe_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,d,e", [(81, 260, 512), (399, 2044, 103), (107, 2048, 384), (10241, 4, 4), (1242, 132, 33)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16"])
def test_many_tokens_equal_few(cuda, t, d, e, dtype):
    torch = cuda
    gen = torch.Generator(device="cuda")
    gen.manual_seed(t)
    x = torch.randn((t, d), device="cuda", generator=gen).to(getattr(torch, dtype))
    w = torch.randn((e, d), device="cuda", generator=gen)
    bias = torch.randn(e, device="cuda", generator=gen) if t % 2 else None
    many = moe_ops.router_logits_t(x, w, bias)
    step = min(8, 40959 // e)
    few = torch.cat([moe_ops.router_logits_t(x[i:i + step].contiguous(), w, bias) for i in range(0, t, step)])
    assert torch.equal(many, few)
    xd, wd = x.double(), w.double()
    ref = xd @ wd.t() + (bias.double() if bias is not None else 0.0)
    scale = xd.abs() @ wd.abs().t() + (bias.double().abs() if bias is not None else 0.0)
    assert ((many.double() - ref).abs() <= scale * (d / 32 + 7) * 2.0 ** -24).all()
    odd = torch.empty(t * d + 1, dtype=x.dtype, device="cuda")[1:].view(t, d)
    odd.copy_(x)
    assert torch.equal(moe_ops.router_logits_t(odd, w, bias), many)


@pytest.mark.parametrize("t", [65535 * 8, 65535 * 8 + 1])
def test_the_largest_batches(cuda, t):
    torch = cuda
    x, w = torch.randn((t, 4), device="cuda"), torch.randn((1, 4), device="cuda")
    got = moe_ops.router_logits_t(x, w).double()
    ref, scale = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert ((got - ref).abs() <= scale * 7 * 2.0 ** -24).all()
