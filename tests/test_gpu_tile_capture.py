"""A captured filter keeps the operator's packed weights: a call that runs out of memory must not take them back."""
import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import _capi as capi
from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu
MB = 1 << 20


def test_weights_of_a_captured_filter_stay():
    import torch
    s, degree = 24, 12
    rp, ci, v = problems.small_laplacian((96, 96, 96), seed=1).csr()
    n = len(rp) - 1
    stream = torch.cuda.Stream()
    ctx = R.Context(0)
    ctx.set_stream(stream.cuda_stream)
    op = R.CsrOperator(ctx, rp, ci, v)
    V0 = torch.randn((s, n), device="cuda", dtype=torch.float64)
    V = V0.clone()
    torch.cuda.synchronize()
    for _ in range(3):  # the weights are laid out in these
        V.copy_(V0)
        torch.cuda.synchronize()
        R.filter_block(ctx, op, V, s, degree, -0.1, 1.9)
        ctx.synchronize()
    want, held = V.clone(), ctx.device_bytes()
    assert ctx.counter("tile_launches") > degree
    graph = torch.cuda.CUDAGraph()
    before = ctx.counter("tile_launches")
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        R.filter_block(ctx, op, V, s, degree, -0.1, 1.9)
    assert ctx.counter("tile_launches") > before
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - 40 * MB, device="cuda", dtype=torch.uint8)
    with pytest.raises(capi.RCError):  # 49 MB of values; the weights are 57 MB
        R.CsrOperator(ctx, rp, ci, v)
    assert ctx.device_bytes() == held
    del ballast
    torch.cuda.empty_cache()
    V.copy_(V0)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(V, want)
    del graph
    op.close()
    ctx.close()
