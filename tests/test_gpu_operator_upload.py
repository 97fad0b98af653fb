"""Operators are complete when they are handed out: their arrays come from pageable host memory through the default
stream, and the context's own stream, which does not wait for that one, reads them at once."""
import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("form", ["csr", "csr without a grid", "stencil"])
@pytest.mark.parametrize("dims", [(3, 4, 5), (40, 30, 20), (96, 80, 64)])
def test_the_first_product_reads_the_whole_operator(form, complex_, dims):
    """Every operator is new and used at once: A v for a block of ones, a sum of at most 7 entries of absolute value at
    most 11, and two steps of the row-major filter (three such sums, each rounded a few times)."""
    import torch
    n = int(np.prod(dims))
    P = problems.small_laplacian(dims, seed=1, complex_=complex_, flux=0.17)
    rp, ci, v = P.csr()
    want = np.add.reduceat(v, rp[:-1])
    ones = np.ones((8, n), dtype=v.dtype)
    if form == "csr without a grid":  # the rows' entries reversed
        order = np.repeat(rp[:-1] + rp[1:] - 1, np.diff(rp)) - np.arange(rp[-1])
        ci, v = ci[order], v[order]
    ctx = R.Context(0)
    X, Y = torch.from_numpy(ones).cuda(), torch.empty((8, n), device="cuda", dtype=torch.from_numpy(ones).dtype)
    torch.cuda.synchronize()
    for _ in range(4):
        op = R.operator_from_problem(ctx, P, "stencil") if form == "stencil" else R.CsrOperator(ctx, rp, ci, v)
        R.spmm(ctx, op, X, Y, 8)
        ctx.synchronize()
        np.testing.assert_allclose(Y.cpu().numpy(), np.tile(want, (8, 1)), rtol=0, atol=7 * 11 * 2.0 ** -52)
        Y.copy_(X)
        torch.cuda.synchronize()
        R.filter_block(ctx, op, Y, 8, 2, -0.1, 1.9)
        ctx.synchronize()
        x1 = -0.19 * want + 1.9
        x2 = (-0.19 * np.add.reduceat(v * x1[ci], rp[:-1]) + 1.9 * x1 - 1.0) / 3.0
        np.testing.assert_allclose(Y.cpu().numpy(), np.tile(x2, (8, 1)), rtol=0, atol=1e-13)
        op.close()
    ctx.close()
