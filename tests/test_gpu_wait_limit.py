"""A stage in shared memory that never lands (RCB200_LOST_STAGES=1: the kernels take the first one for lost, as after a
wait that ran out, and a CTA's copies in flight are still waited for): all that the kernel forms is NaN, nothing of it is
stale, and the same call on another context is right."""
import os

import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu

FORMS = [("csr", 7, False), ("csr", 7, True), ("stencil", 7, False), ("stencil", 7, True), ("stencil", 27, False)]
DIMS, S = (24, 14, 60), 30  # even: the column-major steps take TMA copies


def _context(**env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update({k: str(v) for k, v in env.items()})
    try:
        return R.Context(0)
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k)
            else:
                os.environ[k] = v


def _operator(ctx, form, kind, complex_, dims=DIMS):
    diag = 6.0 + np.random.default_rng(3).uniform(0, 1, int(np.prod(dims)))
    P = problems.Problem("t", dims, kind, diag, -1.0, 0.13 if complex_ else 0.0, complex_)
    return R.operator_from_problem(ctx, P, form)


def _block(n, s, complex_, offset=0):
    import torch
    flat = torch.randn(s * n + offset, device="cuda", dtype=torch.complex128 if complex_ else torch.float64,
                       generator=torch.Generator("cuda").manual_seed(n))
    torch.cuda.synchronize()
    return flat[offset:].view(s, n)


def _all_nan(X):
    import torch
    parts = torch.view_as_real(X) if X.is_complex() else X
    return bool(torch.isnan(parts).all())


ROW_MAJOR = {
    "filter of 2": lambda ctx, op, V, Y: R.filter_block(ctx, op, V, S, 2, -0.1, 1.9),  # (one step: column-major)
    "filter of 4": lambda ctx, op, V, Y: R.filter_block(ctx, op, V, S, 4, -0.1, 1.9),
    "residual block": lambda ctx, op, V, Y: R.filter_correction(ctx, op, V, S, np.linspace(5, 7, S), 1, -0.1, 1.9),
    "correction of 3": lambda ctx, op, V, Y: R.filter_correction(ctx, op, V, S, np.linspace(5, 7, S), 3, -0.1, 1.9),
}
COLUMN_MAJOR = {"step": lambda ctx, op, V, Y: R.spmm(ctx, op, V, Y, S)}
STEPS = [(name, *f) for name in ROW_MAJOR for f in FORMS]
STEPS += [("step", *f) for f in FORMS if f[1] != 27] + [("step", "stencil", 5, False)]


@pytest.mark.parametrize("name,form,kind,complex_", STEPS)
def test_operator_steps(name, form, kind, complex_):
    import torch
    call = {**ROW_MAJOR, **COLUMN_MAJOR}[name]
    for env in ({"RCB200_LOST_STAGES": 1}, {}):
        ctx = _context(RCB200_TILE=2, **env)
        op = _operator(ctx, form, kind, complex_, DIMS if kind != 5 else (DIMS[0], DIMS[1] * DIMS[2], 1))
        V = _block(op.n, S, complex_)
        Y = torch.zeros_like(V)
        torch.cuda.synchronize()
        call(ctx, op, V, Y)
        ctx.synchronize()
        assert ctx.counter("tile_launches") > 0
        X = Y if name in COLUMN_MAJOR else V
        if env:
            assert _all_nan(X)
        else:
            assert bool(torch.isfinite(torch.view_as_real(X) if complex_ else X).all())
        op.close()
        ctx.close()


@pytest.mark.parametrize("n,s,complex_,offset", [
    (2160, 24, False, 0), (2161, 37, False, 0), (40_001, 96, False, 1), (40_000, 192, False, 0), (30_000, 10, False, 0),
    (2160, 24, True, 0), (20_011, 100, True, 0),
])
def test_products(n, s, complex_, offset):
    """CholeskyQR's Gram matrix and product (a Gram matrix of NaN reads as one of zero columns, which the shifted factor
    accepts; the product then fails by itself)."""
    import torch
    ctx = _context(RCB200_LOST_STAGES=1)
    V = _block(n, s, complex_, offset)
    R.cholqr(ctx, V, n, s, complex_=complex_)
    ctx.synchronize()
    assert _all_nan(V)
    ctx.close()
    ctx = _context()
    V = _block(n, s, complex_, offset)
    R.cholqr(ctx, V, n, s, complex_=complex_)
    ctx.synchronize()
    err = V.conj() @ V.T - torch.eye(s, device="cuda", dtype=V.dtype)
    assert float(err.abs().max()) < 1e-13
    ctx.close()


@pytest.mark.parametrize("complex_", [False, True])
def test_ritz_step(complex_):
    """Rayleigh-Ritz: no eigenvalue, vector or residual of a failed step looks good."""
    import torch
    ctx = _context(RCB200_LOST_STAGES=1, RCB200_TILE=2)
    op = _operator(ctx, "stencil", 7, complex_)
    V = _block(op.n, S, complex_)
    W = torch.zeros_like(V)
    torch.cuda.synchronize()
    evals, res = R.rayleigh_ritz(ctx, op, V, W, S, S)[:2]
    assert np.isnan(evals).any() and np.isnan(res).all()
    assert _all_nan(V) and _all_nan(W)
    op.close()
    ctx.close()
