"""The small eigensolve at the sizes where its cluster of CTAs changes and where its shared memory ends."""
import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("s", [1, 2, 3, 5, 31, 40, 41, 64, 80, 81, 127, 143, 144, 145, 193, 300, 330, 471, 480])
@pytest.mark.parametrize("scale", [1.0, 1e-160, 1e150])
def test_small_eigh_edges(ctx, s, complex_, scale):
    """Nearly diagonal matrices as late Ritz steps have them, and graded ones far from unit scale: eigenvalues to
    1e-14 s of the norm, orthonormal vectors and residuals to the same."""
    if scale != 1.0 and s not in (3, 41, 145, 330):
        pytest.skip("scales at a few sizes")
    rng = np.random.default_rng(s)
    X = rng.standard_normal((s, s)) + (1j * rng.standard_normal((s, s)) if complex_ else 0)
    H = np.diag(np.sort(rng.standard_normal(s))).astype(X.dtype) + 1e-3 * (X + X.conj().T)
    w, Q = R.small_eigh(ctx, H * scale)
    w = w / scale
    ref = np.linalg.eigvalsh(H)
    nrm = np.abs(ref).max()
    tol = 1e-14 * max(s, 10)
    assert np.abs(w - ref).max() < tol * nrm
    assert np.abs(Q.conj().T @ Q - np.eye(s)).max() < tol
    assert np.abs(H @ Q - Q * w).max() < 2 * tol * nrm


def test_not_a_number_ends(ctx):
    """A NaN in the matrix rotates nothing: the call returns at once, with no sweep."""
    H = np.diag(np.arange(1.0, 65.0))
    H[3, 5] = H[5, 3] = np.nan
    R.small_eigh(ctx, H)
    assert ctx.counter("jacobi_sweeps") == 0
