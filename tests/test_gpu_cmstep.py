"""Operator steps on column-major FP64 blocks from shared-memory tiles (RCB200_TILE=2: for every size) against the
gather kernels (RCB200_TILE=0): grids smaller than a tile and cut off on every side, few and many columns, leading
dimensions beyond n, an added block; and the residual norms formed beside them."""
import os

import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu

KINDS = [("csr", 7, False), ("csr", 7, True), ("stencil", 7, False), ("stencil", 7, True), ("stencil", 5, False)]


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


def _operator(ctx, form, kind, complex_, dims):
    n = int(np.prod(dims))
    diag = 6.0 + np.random.default_rng(n).uniform(0, 1, n)
    return R.operator_from_problem(ctx, problems.Problem("t", dims, kind, diag, -1.0, 0.13 if complex_ else 0.0, complex_),
                                   form)


def _block(rng, s, ld, complex_):
    V = rng.standard_normal((s, ld))
    return V + 1j * rng.standard_normal((s, ld)) if complex_ else V


@pytest.mark.parametrize("form,kind,complex_", KINDS)
@pytest.mark.parametrize("dims", [(2, 3, 4), (7, 6, 5), (33, 17, 6), (15, 31, 40), (70, 2, 35), (24, 24, 50)])
@pytest.mark.parametrize("s,pad", [(1, 0), (5, 3), (9, 0), (40, 1)])
def test_tile_step_equals_gather_step(form, kind, complex_, dims, s, pad):
    """The same sums in the same order: the same bits, and nothing written beyond row n."""
    import torch
    if kind == 5:
        dims = (dims[0], dims[1] * dims[2], 1)
    n = int(np.prod(dims))
    rng = np.random.default_rng(s)
    X, Y = _block(rng, s, n + pad, complex_), _block(rng, s, n + pad, complex_)
    out = []
    for tile in (0, 2):
        ctx = _context(tile)
        op = _operator(ctx, form, kind, complex_, dims)
        for beta in (0.0, -0.7):
            Xd, Yd = torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda()
            torch.cuda.synchronize()
            R.spmm(ctx, op, Xd, Yd, s, alpha=1.3, beta=beta, ldx=n + pad, ldy=n + pad)
            ctx.synchronize()
            out.append(Yd.cpu().numpy())
            assert np.array_equal(out[-1][:, n:], Y[:, n:])
        op.close()
        ctx.close()
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[3])


@pytest.mark.parametrize("form,kind,complex_", KINDS)
@pytest.mark.parametrize("dims,s,res_count", [((7, 6, 5), 3, 3), ((33, 17, 6), 20, 0), ((24, 24, 30), 33, 17),
                                              ((15, 31, 40), 48, 48)])
def test_residual_norms_beside_the_step(form, kind, complex_, dims, s, res_count):
    """||A v - lam v|| of the Ritz pairs that come back; sums of n squares: n eps of the norm, and the residual's own
    rounding, 8 terms of eps ||A|| each over the root of n rows (n eps covers both here)."""
    import torch
    if kind == 5:
        dims = (dims[0], dims[1] * dims[2], 1)
    n = int(np.prod(dims))
    V = np.linalg.qr(_block(np.random.default_rng(s), s, n, complex_).T)[0].T.copy()
    ctx = _context(2)
    op = _operator(ctx, form, kind, complex_, dims)
    Vd, Wd = torch.from_numpy(V).cuda(), torch.empty((s, n), device="cuda", dtype=torch.from_numpy(V).dtype)
    torch.cuda.synchronize()
    lam, res, _ = R.rayleigh_ritz(ctx, op, Vd, Wd, s, res_count)
    Vn, Wn = Vd.cpu().numpy(), Wd.cpu().numpy()
    want = np.linalg.norm(Wn - lam[:, None] * Vn, axis=1)[:res_count]
    np.testing.assert_allclose(res, want, rtol=n * 2.0 ** -52, atol=n * 2.0 ** -52)
    op.close()
    ctx.close()
