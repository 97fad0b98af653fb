"""The shared-memory tile kernels of 7- and 27-point operators (RCB200_TILE=2: for every size) against the gather
kernels (RCB200_TILE=0): grids smaller than a tile, tiles cut off on every side, one to several panels of columns."""
import os

import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


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
    P = problems.Problem("t", dims, kind, diag, -1.0 / 26.0 if kind == 27 else -1.0, 0.13 if complex_ else 0.0, complex_)
    return R.operator_from_problem(ctx, P, form)


def _run(tile, make, V, call):
    import torch
    ctx = _context(tile)
    op = make(ctx)
    Vd = torch.from_numpy(V.copy()).cuda()
    torch.cuda.synchronize()
    call(ctx, op, Vd)
    ctx.synchronize()
    out = Vd.cpu().numpy()
    op.close()
    ctx.close()
    return out


@pytest.mark.parametrize("form,kind,complex_", [("csr", 7, False), ("csr", 7, True), ("stencil", 7, False),
                                                ("stencil", 7, True), ("stencil", 27, False)])
@pytest.mark.parametrize("dims", [(2, 3, 4), (7, 6, 5), (16, 8, 9), (33, 17, 6), (15, 31, 40), (64, 3, 11)])
@pytest.mark.parametrize("s", [1, 3, 24, 37, 96, 130])
def test_tile_steps_equal_gather_steps(form, kind, complex_, dims, s):
    """7 points: the same sums in the same order, bit for bit. 27 points: other partial sums; in FP64 a step's error is
    at most 30 eps of the block's largest entry (27 terms of weight 1/26 and the diagonal), over 5 steps of gain at most
    2 each; the correction filter rounds residual-sized terms to 8 bits, one step of which may differ."""
    n = int(np.prod(dims))
    if s > n // 2:
        pytest.skip("block too wide for the grid")
    rng = np.random.default_rng(s)
    V = rng.standard_normal((s, n)) + (1j * rng.standard_normal((s, n)) if complex_ else 0)
    make = lambda ctx: _operator(ctx, form, kind, complex_, dims)  # noqa: E731
    filt = lambda ctx, op, Vd: R.filter_block(ctx, op, Vd, s, 5, -0.1, 1.9)  # noqa: E731
    a, b = _run(0, make, V, filt), _run(2, make, V, filt)
    if kind == 27:
        np.testing.assert_allclose(b, a, rtol=0, atol=32 * 30 * 2.0 ** -52 * np.abs(V).max())
    else:
        assert np.array_equal(a, b)
    # the residual block and the correction steps
    lam = rng.uniform(5.0, 7.0, s)
    corr = lambda ctx, op, Vd: R.filter_correction(ctx, op, Vd, s, lam, 6, -0.1, 1.9)  # noqa: E731
    a, b = _run(0, make, V, corr), _run(2, make, V, corr)
    if kind == 27:
        np.testing.assert_allclose(b, a, rtol=0, atol=2.0 ** -6 * np.abs(a).max())
    else:
        assert np.array_equal(a, b)


@pytest.mark.parametrize("change", ["missing pair", "periodic bond", "rows reversed"])
def test_matrices_that_are_no_grid(change):
    """Seven column offsets but not the rows of a grid: the gather kernels serve them, whatever the switch says."""
    import scipy.sparse as sp
    dims, s = (6, 5, 4), 8
    n = int(np.prod(dims))
    rp, ci, v = problems.stencil_csr(dims, 7, 6.0 + np.random.default_rng(1).uniform(0, 1, n), -1.0)
    A = sp.csr_matrix((v, ci, rp), shape=(n, n)).tolil()
    if change == "missing pair":
        A[40, 41] = A[41, 40] = 0.0
    elif change == "periodic bond":
        A[5, 6] = A[6, 5] = -0.5
    A = A.tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    rp, ci, v = A.indptr, A.indices.copy(), A.data.copy()
    if change == "rows reversed":
        for i in range(n):
            ci[rp[i]:rp[i + 1]] = ci[rp[i]:rp[i + 1]][::-1]
            v[rp[i]:rp[i + 1]] = v[rp[i]:rp[i + 1]][::-1]
    V = np.random.default_rng(2).standard_normal((s, n))
    make = lambda ctx: R.CsrOperator(ctx, rp, ci, v)  # noqa: E731
    call = lambda ctx, op, Vd: R.filter_block(ctx, op, Vd, s, 4, -0.1, 1.9)  # noqa: E731
    a, b = _run(0, make, V, call), _run(2, make, V, call)
    assert np.array_equal(a, b)
    x0, x1 = V.T, -0.19 * (A @ V.T) + 1.9 * V.T
    for _ in range(3):
        x0, x1 = x1, -0.19 * (A @ x1) + 1.9 * x1 - x0
    np.testing.assert_allclose(b, (x1 / 5.0).T, rtol=0, atol=1e-13)


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("dims", [(63, 2, 1), (64, 3, 1), (13, 5, 3), (8, 8, 9)])
@pytest.mark.parametrize("s", [1, 9, 32, 33, 70])
def test_correction_exit_is_the_same_for_every_alignment(ctx, complex_, dims, s):
    """The last step reads and writes pairs of rows where they are 16-byte aligned: even and odd leading dimensions and a
    block that starts one entry off give the same bits, and nothing outside the block changes."""
    import torch
    kind = 5 if dims[2] == 1 else 7
    n = int(np.prod(dims))
    op = _operator(ctx, "stencil", kind, complex_, dims)
    rng = np.random.default_rng(s)
    V = rng.standard_normal((s, n)) + (1j * rng.standard_normal((s, n)) if complex_ else 0)
    lam = rng.uniform(5.0, 7.0, s)
    out = []
    for pad, shift in ((0, 0), (1, 0), (2, 1)):
        ld = n + pad
        buf = torch.full((s * ld + 8,), 7.5, dtype=torch.complex128 if complex_ else torch.float64, device="cuda")
        Vd = buf[shift:shift + s * ld].view(s, ld)
        Vd[:, :n] = torch.from_numpy(V)
        torch.cuda.synchronize()
        R.filter_correction(ctx, op, Vd, s, lam, 4, -0.1, 1.9, ld=ld)
        ctx.synchronize()
        out.append(Vd[:, :n].cpu().numpy())
        Vd[:, :n] = 7.5
        assert (buf == 7.5).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    op.close()
