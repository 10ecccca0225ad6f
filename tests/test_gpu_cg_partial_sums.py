"""CG on the loop of separate kernels where the number of partial sums that an
iteration's kernels hand on changes: 1 CTA, the last full CTA of the operator
product (152 of 1024 rows), the last count that the consumer reads in one pass
(160), one more, the widest grid of the vector kernels (304) and rows beyond
it; with the graph loop and with the host loop."""

import numpy as np
import pytest
import scipy.sparse as ss
import torch

from gpu_helpers import to_bsr, vec

pytestmark = pytest.mark.gpu

CTA = 1024


@pytest.mark.parametrize("n", [1, 31, CTA, CTA + 1, 152 * CTA, 152 * CTA + 1, 160 * CTA,
                               160 * CTA + 1, 304 * CTA, 304 * CTA + 33])
@pytest.mark.parametrize("jacobi", [False, True])
def test_partial_sums(n, jacobi):
    from warp_preconditioners_gb300 import SparseOperator
    from warp_preconditioners_gb300.linear import Solver

    rng = np.random.default_rng(n)
    d = 4.0 + rng.uniform(0.0, 1.0, n)
    a = ss.diags([d, -np.ones(max(n - 1, 0)), -np.ones(max(n - 1, 0))], [0, 1, -1]).tocsr()
    b = rng.normal(size=n)
    bnorm = np.linalg.norm(b)
    A = SparseOperator(to_bsr(a))
    M = SparseOperator(to_bsr(ss.diags(1.0 / d).tocsr())) if jacobi else None

    # |A^-1| <= 1/2 (Gershgorin), so |x - A^-1 b| <= |b - A x| / 2; the
    # recursive residual the stop looks at drifts from the true one by less
    # than 100 iterations' rounding, 1e-12 |b|.
    tol = 1e-10
    runs = []
    for graph in (True, False):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        hist = torch.full((200,), -1.0, dtype=torch.float64, device="cuda")
        s = Solver("cg", A, M, use_cuda_graph=graph)
        nit, rr, _ = s.run(vec(b), x, tol=tol, maxiter=100, history=hist)
        k = int(nit.item())
        h = hist.cpu().numpy()
        xs = x.cpu().numpy()
        assert np.linalg.norm(b - a @ xs) <= (tol + 1e-12) * bnorm
        assert h[0] == pytest.approx(bnorm, rel=1e-14)
        assert h[k] == pytest.approx(float(np.sqrt(rr.item())), rel=1e-14)
        assert h[k] <= tol * bnorm * (1 + 1e-12) and (h[:k] > tol * bnorm * (1 - 1e-12)).all()
        assert (h[k + 1:] == -1.0).all()
        runs.append((k, h, xs, s.cluster_size))
    # One iteration limit, on both loops: maxiter stops the count and the state.
    for graph in (True, False):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        nit, _, _ = Solver("cg", A, M, use_cuda_graph=graph).run(vec(b), x, tol=0.0, maxiter=3)
        assert int(nit.item()) <= 3
    if runs[0][3] == 0:  # the same kernels on both loops: the same bits
        assert runs[0][0] == runs[1][0]
        np.testing.assert_array_equal(runs[0][1], runs[1][1])
        np.testing.assert_array_equal(runs[0][2], runs[1][2])
