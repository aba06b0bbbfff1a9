"""The benchmark's own measurement of the grouped gate/up launches, on a small stack."""

import pytest

import bench
from mylocal_llm_b200.moe_stack import PackedMoEStack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 40])
def test_every_gate_up_launch_of_a_step_is_timed(cuda, tokens):
    torch = cuda
    stack = PackedMoEStack.synthetic(3, d_model=512, d_ff=256, n_experts=16, top_k=4, shared_d_ff=256, seed=1)
    x = torch.randn((1, tokens, 512), device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        records = bench.gate_up_records(torch, stream, stack, lambda: stack.forward(x)[0])
    assert len(records) == 3
    for start, end, counts in records:
        assert start.elapsed_time(end) > 0 and int(counts.sum()) == tokens * 5
    assert stack.persistent_step
