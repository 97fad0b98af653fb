"""Operator steps on column-major blocks of grids a few points wide, where most of a tile would lie outside the grid: by
default the gather kernels serve them. The tiles show in the scratch of a Rayleigh-Ritz step (their residual norms have
one partial sum per tile and column, and CSR rows their packed weights)."""
import os

import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


def _scratch(tile, form, kind, complex_, dims, s):
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
    diag = 6.0 + np.random.default_rng(n).uniform(0, 1, n)
    P = problems.Problem("t", dims, kind, diag, -1.0, 0.13 if complex_ else 0.0, complex_)
    op = R.operator_from_problem(ctx, P, form)
    V = torch.randn((s, n), device="cuda", dtype=torch.complex128 if complex_ else torch.float64)
    W = torch.empty_like(V)
    torch.cuda.synchronize()
    R.cholqr(ctx, V, n, s, complex_)
    R.rayleigh_ritz(ctx, op, V, W, s, s)
    used = ctx.device_bytes()
    op.close()
    ctx.close()
    return used


@pytest.mark.parametrize("form,kind,complex_,dims,s", [
    ("csr", 7, False, (2, 2, 200000), 96), ("csr", 7, True, (2, 2, 200000), 56), ("stencil", 7, False, (2, 2, 200000), 96),
    ("stencil", 7, True, (2, 2, 200000), 56), ("csr", 7, False, (8, 8, 13001), 96), ("stencil", 5, False, (2, 600000, 1), 96)])
def test_narrow_grids_take_the_gather_kernels(form, kind, complex_, dims, s):
    assert _scratch(1, form, kind, complex_, dims, s) == _scratch(0, form, kind, complex_, dims, s)


@pytest.mark.parametrize("form,kind,complex_", [("csr", 7, False), ("csr", 7, True), ("stencil", 7, False)])
def test_wide_grids_take_the_tiles(form, kind, complex_):
    dims, s = (128, 96, 64), 96 if not complex_ else 64
    used = _scratch(1, form, kind, complex_, dims, s)
    assert used == _scratch(2, form, kind, complex_, dims, s)
    if form == "csr":
        assert used > _scratch(0, form, kind, complex_, dims, s)
