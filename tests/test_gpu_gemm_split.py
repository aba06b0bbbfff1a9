"""Split of K in the tensor-core GEMM where the 256-position groups are no power of two, or the row count no multiple of
four: uneven parts, a last part of one group, 33 groups (eight parts would leave the last one empty), partial sums of an
odd length. Bars of ``test_gpu_gemm.check``: FP64 over BF16-rounded and over exact weights."""

import pytest

from mylocal_llm_b200.quantize import random_packed
from test_gpu_gemm import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,n,k,m", [("Q6_K", 203, 2816, 77), ("Q4_K", 130, 8448, 20), ("Q5_K", 33, 2304, 33),
                                       ("Q8_0", 1001, 3328, 257), ("Q6_K", 5, 2048, 19), ("Q4_K", 127, 5120, 513)])
@pytest.mark.parametrize("out", ["float32", "bfloat16"])
def test_uneven_parts(cuda, fmt, n, k, m, out):
    check(cuda, random_packed(fmt, (n, k), seed=n, d=0.01, dmin=0.005), m, seed=m, out_dtype=getattr(cuda, out), split=True)
