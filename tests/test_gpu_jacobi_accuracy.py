"""The rotations of the small eigensolve are unitary to the last bit: no drift of the columns' lengths."""
import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("s,matrices", [(24, 20), (41, 12), (96, 6)])
def test_columns_keep_their_length(ctx, s, matrices, complex_):
    """A column sees about 5 sweeps of s rotations. Unbiased roundings leave its squared norm off by about
    eps sqrt(5 s), and the mean over s columns of N matrices by eps sqrt(5 / N): at most three times that. A cosine that
    is systematically an ulp low leaves 5 eps and more (s = 24)."""
    mean = 0.0
    for k in range(matrices):
        rng = np.random.default_rng(100 * s + k)
        X = rng.standard_normal((s, s)) + (1j * rng.standard_normal((s, s)) if complex_ else 0)
        H = np.diag(np.sort(rng.standard_normal(s))).astype(X.dtype) + 1e-2 * (X + X.conj().T)
        _, Q = R.small_eigh(ctx, H)
        q = np.stack([Q.real, Q.imag]).astype(np.longdouble)
        mean += float(((q ** 2).sum(axis=(0, 1)) - 1).mean()) / matrices
    assert abs(mean) < 3 * np.sqrt(5 / matrices) * EPS
