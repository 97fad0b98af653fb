"""The small eigensolve where no cluster holds the matrix: the grid kernel's barrier words lie between the eigenvalues
and the eigenvectors, whose distance is a multiple of 256 bytes. At s = 31 mod 32 the eigenvalues and two words fill it
to the last byte, so a third word would be the first entry of Q."""
import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,complex_", [(479, False), (511, False), (351, True), (383, True)])
def test_barrier_words_do_not_touch_the_vectors(ctx, s, complex_):
    """A diagonal matrix: Q is a permutation and Q[0, 0] one, the bits that would read as "give up"; and a nearly
    diagonal one to the bounds of the other sizes (1e-14 s of the norm)."""
    d = np.sort(np.random.default_rng(s).standard_normal(s))
    dt = np.complex128 if complex_ else np.float64
    w, Q = R.small_eigh(ctx, np.diag(d).astype(dt))
    assert np.array_equal(w, d) and np.array_equal(Q, np.eye(s, dtype=dt))
    rng = np.random.default_rng(1)
    X = rng.standard_normal((s, s)) + (1j * rng.standard_normal((s, s)) if complex_ else 0)
    H = np.diag(d).astype(dt) + 1e-3 * (X + X.conj().T)
    w, Q = R.small_eigh(ctx, H)
    ref = np.linalg.eigvalsh(H)
    tol = 1e-14 * s
    assert np.abs(w - ref).max() < tol * np.abs(ref).max()
    assert np.abs(Q.conj().T @ Q - np.eye(s)).max() < tol
    assert np.abs(H @ Q - Q * w).max() < 2 * tol * np.abs(ref).max()
