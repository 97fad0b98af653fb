"""The small eigensolve of one CTA (RCB200_JACOBI_CTAS=1) with a table of a round's rotations beyond the 48 KB of shared
memory that a launch gets by itself: real from 3073, complex from 2458 rows. Diagonal matrices, which take no rotation."""
import os

import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,complex_", [(3100, False), (2500, True)])
def test_rotations_beyond_48_kb(s, complex_):
    old = os.environ.get("RCB200_JACOBI_CTAS")
    os.environ["RCB200_JACOBI_CTAS"] = "1"
    try:
        ctx = R.Context(0)
    finally:
        if old is None:
            os.environ.pop("RCB200_JACOBI_CTAS")
        else:
            os.environ["RCB200_JACOBI_CTAS"] = old
    d = np.random.default_rng(s).standard_normal(s)
    w, Q = R.small_eigh(ctx, np.diag(d).astype(np.complex128 if complex_ else np.float64))
    order = np.argsort(d)
    assert np.array_equal(w, d[order])
    want = np.zeros((s, s))
    want[order, np.arange(s)] = 1.0
    assert np.array_equal(Q, want)
    ctx.close()
