"""The batch runner that a context keeps between calls of the batched correction filter: calls in a row, with other
blocks and job counts (its table slots come round), and contexts that go away in between."""
import numpy as np
import pytest

from rayleighchebyshevgpgpu_b200 import problems
from rayleighchebyshevgpgpu_b200 import runtime as R

pytestmark = pytest.mark.gpu


def test_calls_in_a_row_give_the_bits_of_new_contexts():
    import torch
    P = problems.small_laplacian((12, 9, 7), seed=3)
    rng = np.random.default_rng(0)
    blocks = [[(rng.standard_normal((s, P.n)), rng.uniform(5.0, 7.0, s)) for s in sizes]
              for sizes in ((8, 3), (16,), (5, 24, 7), (8, 3), (1, 2, 3, 4), (40,), (9, 9))]

    def run(ctx, op, jobs):
        Vd = [torch.from_numpy(V).cuda() for V, _ in jobs]
        torch.cuda.synchronize()
        got = R.filter_correction_batch(ctx, [(op, v, v.shape[0], lam, 6, -0.1, 1.9) for v, (_, lam) in zip(Vd, jobs)])
        return got, [v.cpu().numpy() for v in Vd]

    kept = R.Context(0)
    op = R.operator_from_problem(kept, P, "csr")
    for jobs in blocks:
        got, out = run(kept, op, jobs)
        fresh = R.Context(0)
        op2 = R.operator_from_problem(fresh, P, "csr")
        want_got, want = run(fresh, op2, jobs)
        op2.close()
        fresh.close()
        assert got == want_got
        for a, b in zip(out, want):
            assert np.array_equal(a, b)
    op.close()
    kept.close()
