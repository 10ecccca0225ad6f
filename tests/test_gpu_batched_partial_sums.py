"""Batched CG where the number of partial sums of a dot product changes: one,
as many as there are groups (16) and one more, the CTAs that are resident at
once (304) and one more, one short of the cap (608), the cap and rows beyond
it; with full and ragged groups of right-hand sides."""

import numpy as np
import pytest
import scipy.sparse as ss
import torch

from gpu_helpers import to_bsr, vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3, 20, 32])
@pytest.mark.parametrize("parts,extra", [(0, 1), (16, 0), (16, 1), (304, 0), (304, 1), (607, 0),
                                         (608, 0), (608, 5), (1700, 3)])
def test_partial_sums(k, parts, extra):
    from warp_preconditioners_gb300 import SparseOperator, batched

    lanes = 1 << (k - 1).bit_length()
    n = parts * 16 * (32 // lanes) + extra
    rng = np.random.default_rng(100 * k + parts + extra)
    d = 4.0 + rng.uniform(0.0, 1.0, n)
    off = -np.ones(n - 1)
    a = ss.diags([d, off, off], [0, 1, -1]).tocsr()
    b = rng.normal(size=(n, k))
    b[:, k // 2] *= 1e-3
    A = to_bsr(a)
    M = to_bsr(ss.diags(1.0 / d).tocsr())
    solver = batched.BatchedCG(batched.batched_sparse(A), batched.batched_sparse(M))

    # |A^-1| <= 1/2 (Gershgorin); the recursive residual the stop looks at
    # drifts from the true one by less than 100 iterations' rounding.
    tol = 1e-10
    out = []
    for _ in range(2):
        X = torch.zeros((n, k), dtype=torch.float64, device="cuda")
        nit, rr = solver.run(vec(b), X, tol=tol, maxiter=100)
        out.append((nit.cpu().numpy().copy(), rr.cpu().numpy().copy(), X.cpu().numpy()))
    x = out[0][2]
    bnorm = np.linalg.norm(b, axis=0)
    res = np.linalg.norm(b - a @ x, axis=0)
    assert (res <= (tol + 1e-12) * bnorm).all()
    assert (np.sqrt(out[0][1][:k]) <= tol * bnorm * (1 + 1e-12)).all()
    assert (out[0][0][:k] < 100).all()
    for one, two in zip(out[0], out[1]):
        np.testing.assert_array_equal(one, two)
