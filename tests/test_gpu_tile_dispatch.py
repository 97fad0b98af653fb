"""The tile kernels as large blocks run them, every CTA with several units one after the other (the ring's slots and
phases and the residual's column sums carried on from one to the next), and the default switch on both sides of its
lines: against the gather kernels (RCB200_TILE=0)."""
import os

import numpy as np
import pytest

from oracle import rc_oracle as O
from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu

FORMS = [("csr", 7, False), ("csr", 7, True), ("stencil", 7, False), ("stencil", 7, True), ("stencil", 27, False)]
# 396 to 1584 units of tiles for 148 CTAs, cut off on two sides
DIMS, S = (130, 70, 20), 96


def _context(tile):
    old = os.environ.get("RCB200_TILE")
    os.environ["RCB200_TILE"] = str(tile)
    try:
        return R.Context(0)
    finally:
        if old is None:
            os.environ.pop("RCB200_TILE", None)
        else:
            os.environ["RCB200_TILE"] = old


def _problem(kind, complex_, dims):
    n = int(np.prod(dims))
    diag = 6.0 + np.random.default_rng(n).uniform(0, 1, n)
    return problems.Problem("t", dims, kind, diag, -1.0 / 26.0 if kind == 27 else -1.0, 0.13 if complex_ else 0.0, complex_)


def _run(tile, form, kind, complex_, dims, s, call, times=1):
    """The block after `call`, and the launches from tiles, of the last of several calls."""
    import torch
    ctx = _context(tile)
    op = R.operator_from_problem(ctx, _problem(kind, complex_, dims), form)
    V0 = torch.randn((s, op.n), device="cuda", dtype=torch.complex128 if complex_ else torch.float64,
                     generator=torch.Generator("cuda").manual_seed(s))
    for _ in range(times):
        before = ctx.counter("tile_launches")
        V = V0.clone()
        torch.cuda.synchronize()
        call(ctx, op, V)
        ctx.synchronize()
    launches = ctx.counter("tile_launches") - before
    op.close()
    ctx.close()
    return V, launches


@pytest.mark.parametrize("form,kind,complex_", FORMS)
def test_filter_of_several_units(form, kind, complex_):
    """7 points: bit for bit. 27: 5 steps of gain at most 2, each off by at most 30 eps of the largest entry."""
    import torch
    call = lambda ctx, op, V: R.filter_block(ctx, op, V, S, 5, -0.1, 1.9)  # noqa: E731
    want, none = _run(0, form, kind, complex_, DIMS, S, call)
    assert none == 0
    for tile in (1, 2):
        got, launches = _run(tile, form, kind, complex_, DIMS, S, call)
        assert launches == 5 if tile == 2 else launches >= 3  # (by default not the first, and CSR rows later)
        if kind == 27:
            assert float((got - want).abs().max()) <= 32 * 30 * 2.0 ** -52 * float(want.abs().max())
        else:
            assert torch.equal(got, want)


@pytest.mark.parametrize("form,kind,complex_", FORMS)
def test_correction_of_several_units(form, kind, complex_):
    """The residual block and 2 steps with a source. 7 points: bit for bit. 27: FP32 sums in another order move an entry
    to the next bfloat16 (2^-8 of it) with a chance of 4e-4 a step, and such an entry moves about as many neighbours in
    the next: less than 1 % of the entries, 4e-4 of the block's root mean square. (A neighbour left out is 4e-3 of it.)"""
    import torch
    lam = np.random.default_rng(S).uniform(5.0, 7.0, S)
    call = lambda ctx, op, V: R.filter_correction(ctx, op, V, S, lam, 3, -0.1, 1.9)  # noqa: E731
    want, none = _run(0, form, kind, complex_, DIMS, S, call)
    assert none == 0
    for tile in (1, 2):
        # (the CSR rows' weights are laid out in the first calls)
        got, launches = _run(tile, form, kind, complex_, DIMS, S, call, times=5 if tile == 1 else 1)
        assert launches == 3 if tile == 2 else launches >= 2
        if kind == 27:
            d = (got - want).abs()
            assert float((d > 1e-5 * want.abs().mean()).double().mean()) < 1e-2
            assert float(d.square().mean().sqrt()) <= 4e-4 * float(want.square().mean().sqrt())
        else:
            assert torch.equal(got, want)


@pytest.mark.parametrize("form,kind,complex_", FORMS)
def test_residuals_of_several_units(form, kind, complex_):
    """A few iterations of a solve: the residual norms that come back with the Ritz pairs are those of the pairs (sums of
    n squares, n eps, and the pairs' own rounding)."""
    P = _problem(kind, complex_, DIMS)
    A = O.csr_matrix(*P.csr()) if kind != 27 else None
    for tile in (1, 2):
        ctx = _context(tile)
        op = R.operator_from_problem(ctx, P, form)
        p = R.make_params(64, 5e-2, incr=64, buffer=32)
        res = R.solve(ctx, op, p)
        assert res.info["found"] == 64 and ctx.counter("tile_launches") > 0
        if A is None:
            import torch
            X = torch.from_numpy(res.evecs).cuda()
            Y = torch.empty_like(X)
            torch.cuda.synchronize()
            gather = _context(0)
            op0 = R.operator_from_problem(gather, P, form)
            R.spmm(gather, op0, X, Y, 64)
            gather.synchronize()
            AX = Y.cpu().numpy()
            op0.close()
            gather.close()
        else:
            AX = (A @ res.evecs.T).T
        r = np.linalg.norm(AX - res.evals[:, None] * res.evecs, axis=1)
        assert r.min() > 1e-6
        np.testing.assert_allclose(res.residuals, r, rtol=1e-6)
        op.close()
        ctx.close()


@pytest.mark.parametrize("form,kind,complex_,dims,s,correction,tiles", [
    ("stencil", 7, False, (40, 40, 40), 53, False, 0),       # FP64 blocks below 32 MB
    ("stencil", 7, False, (48, 48, 48), 53, False, 4),
    ("stencil", 7, False, (300, 130, 2), 53, False, 1),      # two planes: the first step only
    ("stencil", 7, False, (18, 11, 4000), 12, False, 0),     # too few threads
    ("stencil", 7, True, (16, 40, 40), 8, False, 0),         # c128 below 16 MB
    ("stencil", 7, True, (32, 32, 32), 53, False, 4),
    ("stencil", 7, False, (32, 32, 32), 24, True, 1),        # bfloat16 below 4 MB: the residual only
    ("stencil", 7, False, (64, 64, 64), 24, True, 4),
    ("stencil", 7, False, (100, 90, 60), 8, True, 1),        # one slice a row
    ("stencil", 7, False, (100, 90, 5), 130, True, 0),       # an empty last turn; the residual's edges
    ("csr", 7, False, (20, 20, 20), 24, False, 0),           # FP64 rows below 4 MB
    ("csr", 7, False, (64, 64, 64), 24, False, 4),
    ("csr", 7, True, (20, 20, 20), 53, False, 0),            # c128 rows below 32 MB
    ("csr", 7, True, (64, 64, 64), 24, False, 4),
    ("csr", 7, False, (64, 64, 64), 24, True, 4),
])
def test_default_switch(form, kind, complex_, dims, s, correction, tiles):
    import torch
    lam = np.linspace(5.0, 7.0, s)
    if correction:
        call = lambda ctx, op, V: R.filter_correction(ctx, op, V, s, lam, 4, -0.1, 1.9)  # noqa: E731
    else:
        call = lambda ctx, op, V: R.filter_block(ctx, op, V, s, 4, -0.1, 1.9)  # noqa: E731
    want, _ = _run(0, form, kind, complex_, dims, s, call)
    got, launches = _run(1, form, kind, complex_, dims, s, call, times=20 if form == "csr" else 1)
    assert torch.equal(got, want)
    assert launches == tiles
