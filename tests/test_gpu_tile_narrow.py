"""27-point grids a few points wide, where most of a tile lies outside the grid: by default the gather kernels serve
them, as they serve blocks with RCB200_TILE=0; wide grids take the tiles (their sums are formed in another order)."""
import os

import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


def _run(tile, dims, s, correction):
    import torch
    old = os.environ.get("RCB200_TILE")
    os.environ["RCB200_TILE"] = str(tile)
    try:
        ctx = R.Context(0)
    finally:
        if old is None:
            os.environ.pop("RCB200_TILE", None)
        else:
            os.environ["RCB200_TILE"] = old
    n = int(np.prod(dims))
    diag = 1.0 + np.random.default_rng(n).uniform(0, 1, n)
    op = R.operator_from_problem(ctx, problems.Problem("t", dims, 27, diag, -1.0 / 26.0, 0.0, False), "stencil")
    V = torch.randn((s, n), device="cuda", dtype=torch.float64, generator=torch.Generator("cuda").manual_seed(s))
    torch.cuda.synchronize()
    if correction:
        R.filter_correction(ctx, op, V, s, np.linspace(0.5, 1.5, s), 5, -0.1, 1.9)
    else:
        R.filter_block(ctx, op, V, s, 5, -0.1, 1.9)
    ctx.synchronize()
    op.close()
    ctx.close()
    return V


@pytest.mark.parametrize("dims,s", [((2, 2, 50000), 8), ((2, 2, 50000), 48), ((3, 5, 60000), 24), ((8, 8, 100000), 3)])
@pytest.mark.parametrize("correction", [False, True])
def test_narrow_grids_take_the_gather_kernels(dims, s, correction):
    import torch
    assert torch.equal(_run(1, dims, s, correction), _run(0, dims, s, correction))


@pytest.mark.parametrize("dims,s", [((2, 2, 2000), 8), ((6, 6, 6000), 96), ((40, 40, 40), 24), ((64, 1, 4000), 24)])
def test_other_grids_take_the_tiles(dims, s):
    import torch
    assert torch.equal(_run(1, dims, s, False), _run(2, dims, s, False))
    assert not torch.equal(_run(1, dims, s, False), _run(0, dims, s, False))
