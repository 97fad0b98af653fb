"""The small Cholesky factor of CholeskyQR in registers (one CTA to 96 columns, a cluster of four to 192): the widths
where its rows per lane and columns per warp change, against the factor of a QR."""
import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("s", [1, 2, 16, 31, 32, 33, 64, 65, 95, 96, 97, 128, 129, 160, 161, 191, 192, 193])
def test_first_pass_factor(ctx, complex_, s):
    """Two passes on columns of very different norms (condition below 100 once scaled): V R^-1 is the QR's Q with a
    positive diagonal; an entry's error is a few s eps."""
    import torch
    n = 4 * s + 3
    rng = np.random.default_rng(s)
    V = rng.standard_normal((s, n)) + (1j * rng.standard_normal((s, n)) if complex_ else 0)
    V *= np.logspace(-3, 3, s)[:, None]
    Vd = torch.from_numpy(V).cuda()
    torch.cuda.synchronize()
    assert R.cholqr(ctx, Vd, n, s, complex_) == 2
    q, r = np.linalg.qr(V.T)
    ph = np.diag(r) / np.abs(np.diag(r))
    np.testing.assert_allclose(Vd.cpu().numpy(), (q * ph).T, rtol=0, atol=1e-13)


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("s", [24, 96, 150])
def test_breakdown_is_shifted(ctx, complex_, s):
    """A column that repeats another to 1e-10: the first factor fails, the shifted ones give an orthonormal basis."""
    import torch
    n = 3000
    rng = np.random.default_rng(s)
    V = rng.standard_normal((s, n)) + (1j * rng.standard_normal((s, n)) if complex_ else 0)
    V[s // 2] = V[0] + 1e-10 * rng.standard_normal(n)
    Vd = torch.from_numpy(V).cuda()
    torch.cuda.synchronize()
    assert R.cholqr(ctx, Vd, n, s, complex_) > 2
    Q = Vd.cpu().numpy()
    np.testing.assert_allclose(Q.conj() @ Q.T, np.eye(s), rtol=0, atol=1e-12)
