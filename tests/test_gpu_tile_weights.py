"""A CSR operator's packed weights for the tile kernels only save time: they are laid out when the steps have work for
them, and nothing is refused for their sake."""
import os
import re

import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import _capi as capi
from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu
MB = 1 << 20


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


def _matrix(dims, complex_=False):
    """CSR arrays of a grid, and of the same matrix with the rows' entries reversed (no grid to the library)."""
    rp, ci, v = problems.small_laplacian(dims, seed=1, complex_=complex_, flux=0.1).csr()
    order = np.repeat(rp[:-1] + rp[1:] - 1, np.diff(rp)) - np.arange(rp[-1])
    return rp, (ci, v), (ci[order], v[order])


@pytest.mark.parametrize("complex_", [False, True])
def test_a_new_operator_holds_its_arrays_only(complex_):
    import torch
    rp, grid, other = _matrix((40, 30, 20), complex_)
    n, used = len(rp) - 1, []
    for ci, v in (grid, other):
        ctx = R.Context(0)
        op = R.CsrOperator(ctx, rp, ci, v)
        used.append(ctx.device_bytes())
        V = torch.randn((8, n), device="cuda", dtype=torch.complex128 if complex_ else torch.float64)
        torch.cuda.synchronize()
        R.filter_block(ctx, op, V, 8, 4, -0.1, 1.9)
        R.filter_correction(ctx, op, V, 8, np.linspace(5, 7, 8), 4, -0.1, 1.9)
        used.append(ctx.device_bytes())
        op.close()
        ctx.close()
    assert used[0] == used[2] and used[1] == used[3]


def test_the_server_charges_the_arrays_only():
    """Also once calls outside the server have had the weights laid out."""
    import torch
    rp, grid, other = _matrix((40, 30, 20))
    n, need = len(rp) - 1, []
    for ci, v in (grid, other):
        ctx = _context(2)
        op = R.CsrOperator(ctx, rp, ci, v)
        V = torch.randn((8, n), device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        R.filter_block(ctx, op, V, 8, 4, -0.1, 1.9)
        ctx.synchronize()
        with R.Server(0, max_active=1, budget_bytes=MB) as srv:
            with pytest.raises(capi.RCError) as e:
                srv.submit(op, R.make_params(8, 1e-8, buffer=8))
            need.append(int(re.search(r"needs (\d+) device bytes", str(e.value)).group(1)))
        op.close()
        ctx.close()
    assert need[0] == need[1]


def test_short_memory_refuses_nothing():
    """A grid of 2 million rows, 134 MB of weights: with 60 MB more than its arrays take the operator is made and used
    without them; and weights that are there are given back to a call that needs the room."""
    import torch
    dims, s = (128, 128, 128), 8
    n = 128 ** 3
    rp, (ci, v), _ = _matrix(dims)
    want = np.add.reduceat(v, rp[:-1])
    X = torch.ones((s, n), device="cuda", dtype=torch.float64)
    Y = torch.empty_like(X)
    ctx = _context(2)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()

    def fill(leave):
        torch.cuda.synchronize()
        return torch.empty(torch.cuda.mem_get_info()[0] - leave, device="cuda", dtype=torch.uint8)

    def product(op):
        Y.zero_()
        torch.cuda.synchronize()
        R.spmm(ctx, op, X, Y, s)
        ctx.synchronize()
        # sums of 7 entries of absolute value at most 11
        np.testing.assert_allclose(Y[s - 1].cpu().numpy(), want, rtol=0, atol=7 * 11 * 2.0 ** -52)

    ballast = fill(rp.nbytes + ci.nbytes + v.nbytes + 60 * MB)
    op = R.CsrOperator(ctx, rp, ci, v)
    product(op)
    assert ctx.device_bytes() < rp.nbytes + ci.nbytes + v.nbytes + MB
    op.close()
    del ballast
    torch.cuda.empty_cache()

    op = R.CsrOperator(ctx, rp, ci, v)
    product(op)
    assert ctx.device_bytes() >= rp.nbytes + ci.nbytes + v.nbytes + n * 64
    V = torch.randn((s, n), device="cuda", dtype=torch.float64)
    ballast = fill(90 * MB)
    R.cholqr(ctx, V, n, s)  # 134 MB of scratch
    assert abs(float(torch.dot(V[0], V[s - 1]))) < 1e-13 and abs(float(torch.dot(V[0], V[0])) - 1) < 1e-13
    product(op)
    del ballast
    torch.cuda.empty_cache()
    op.close()
    ctx.close()


@pytest.mark.parametrize("complex_,s", [(False, 96), (True, 40)])
def test_the_same_bits_before_and_after(complex_, s):
    """The default switch on 64^3 rows: the weights come in the middle of these calls."""
    import torch
    rp, (ci, v), _ = _matrix((64, 64, 64), complex_)
    n, out = len(rp) - 1, []
    V0 = torch.randn((s, n), device="cuda", dtype=torch.complex128 if complex_ else torch.float64)
    for tile in (0, 1):
        ctx = _context(tile)
        op = R.CsrOperator(ctx, rp, ci, v)
        for _ in range(3):
            V = V0.clone()
            torch.cuda.synchronize()
            R.filter_block(ctx, op, V, s, 8, -0.1, 1.9)
            R.filter_correction(ctx, op, V, s, np.linspace(5, 7, s), 16, -0.1, 1.9)
            W = torch.empty_like(V)
            R.spmm(ctx, op, V, W, s)
            ctx.synchronize()
            out.append((V, W))
        grown = ctx.device_bytes()
        op.close()
        grown -= ctx.device_bytes()
        size = 2 if complex_ else 1
        assert (grown >= rp.nbytes + ci.nbytes + v.nbytes + v.nbytes // 2 + 64 * size * n) == (tile == 1)
        ctx.close()
    for V, W in out[1:]:
        assert torch.equal(V, out[0][0]) and torch.equal(W, out[0][1])
