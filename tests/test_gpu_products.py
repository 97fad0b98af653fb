"""The tall-skinny products behind orthonormalisation and the Ritz step, at the sizes where their tiles, column
groups and alignment cases end: against the same product in numpy."""
import numpy as np
import pytest

from oracle import rc_oracle as O
from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("dims,s,pad", [
    ((33, 1), 1, 0),            # one column, one ragged row tile
    ((257, 1), 7, 0),           # odd leading dimension, odd width
    ((64, 9), 24, 1),           # rows a multiple of the tile, leading dimension made odd
    ((41, 25), 33, 0),          # odd rows, odd width
    ((50, 41), 48, 2),          # one column group filled
    ((61, 71), 49, 0),          # just past it
    ((97, 83), 96, 0),          # two column groups, odd rows
    ((64, 64), 97, 0),          # just past them
    ((53, 29), 192, 1),         # all columns of one pass
    ((47, 31), 193, 0),         # two passes: not in place
])
def test_ritz_vectors_are_the_product_with_q(ctx, complex_, dims, s, pad):
    """V_out = V Q, W = A V_out and the residuals, from the Q that the call returns. Rows of V have norm at most 1
    and so have columns of Q: an entry's rounding error is at most 2 s eps."""
    import torch
    P = problems.small_laplacian(dims, seed=5, complex_=complex_, flux=0.21)
    rng = np.random.default_rng(s)
    X = rng.standard_normal((P.n, s)) + (1j * rng.standard_normal((P.n, s)) if complex_ else 0)
    V = np.linalg.qr(X)[0].T
    ld = P.n + pad
    Vd = torch.zeros((s, ld), dtype=torch.complex128 if complex_ else torch.float64, device="cuda")
    Wd = torch.full_like(Vd, 3.25)
    Vd[:, :P.n] = torch.from_numpy(np.ascontiguousarray(V))
    Vd[:, P.n:] = 7.5
    op = R.operator_from_problem(ctx, P, "csr")
    torch.cuda.synchronize()
    w, res, Q = R.rayleigh_ritz(ctx, op, Vd, Wd, s, s, ld=ld)
    out, W = Vd.cpu().numpy(), Wd.cpu().numpy()
    assert (out[:, P.n:] == 7.5).all() and (W[:, P.n:] == 3.25).all()
    out, W = out[:, :P.n], W[:, :P.n]
    np.testing.assert_allclose(out, Q.T @ V, rtol=0, atol=(8 if complex_ else 4) * s * EPS)
    A = O.csr_matrix(*P.csr())
    AV = (A @ out.T).T
    np.testing.assert_allclose(W, AV, rtol=0, atol=200 * EPS)
    np.testing.assert_allclose(res, np.linalg.norm(AV - w[:, None] * out, axis=1), rtol=0, atol=1e-12)


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("s", [1, 7, 8, 9, 17, 25, 33, 41, 49, 64, 65, 81, 96, 97, 129, 161, 192])
@pytest.mark.parametrize("n,pad,shift", [(0, 0, 0), (1037, 0, 0), (1037, 1, 0), (20000, 1, 0), (1031, 2, 1)])
def test_gram_tiles(ctx, complex_, s, n, pad, shift):
    """Cholesky QR at every number of 8-column tiles, the fewest rows (n = s), leading dimensions even and odd, and
    blocks that start 8 bytes (a complex entry) off: the factor of a QR with a positive diagonal. Two passes from a
    random block (condition below 1e3 for n > s): an entry's error is a few s eps."""
    import torch
    rng = np.random.default_rng(100 * s + n)
    n = n or s
    V = rng.standard_normal((s, n)) + (1j * rng.standard_normal((s, n)) if complex_ else 0)
    if n == s:
        V += 4 * s * np.eye(s)
    ld = n + pad
    buf = torch.zeros(s * ld + 8, dtype=torch.complex128 if complex_ else torch.float64, device="cuda")
    Vd = buf[shift:shift + s * ld].view(s, ld)
    Vd[:, :n] = torch.from_numpy(V)
    torch.cuda.synchronize()
    R.cholqr(ctx, Vd, n, s, complex_, ld=ld)
    out = Vd.cpu().numpy()
    assert not out[:, n:].any()
    q, r = np.linalg.qr(V.T)
    ph = np.diag(r) / np.abs(np.diag(r))
    np.testing.assert_allclose(out[:, :n], (q * ph).T, rtol=0, atol=1e-13)


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("s,n,pad", [(193, 1500, 0), (217, 1501, 0), (385, 2000, 1)])
def test_triangular_products_in_several_passes(ctx, complex_, s, n, pad):
    """Products with an upper triangular T of more than 192 columns: a pass's first tiles end far down in T."""
    import torch
    rng = np.random.default_rng(s)
    V = rng.standard_normal((s, n)) + (1j * rng.standard_normal((s, n)) if complex_ else 0)
    Vd = torch.zeros((s, n + pad), dtype=torch.complex128 if complex_ else torch.float64, device="cuda")
    Vd[:, :n] = torch.from_numpy(V)
    torch.cuda.synchronize()
    R.cholqr(ctx, Vd, n, s, complex_, ld=n + pad)
    q, r = np.linalg.qr(V.T)
    ph = np.diag(r) / np.abs(np.diag(r))
    np.testing.assert_allclose(Vd.cpu().numpy()[:, :n], (q * ph).T, rtol=0, atol=1e-13)
