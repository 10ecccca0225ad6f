"""GMRES at basis sizes around the chunks of 16 vectors, with one row, less and
more rows than the dot products' threads, against the textbook oracle."""

import numpy as np
import pytest
import scipy.sparse as ss
import torch

from gpu_helpers import oracle_csr, to_bsr, vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 257, 3000, 77824, 90001])
@pytest.mark.parametrize("restart,steps", [(1, 4), (15, 15), (16, 16), (17, 35), (32, 32), (33, 33),
                                           (64, 64)])
def test_basis_sizes(oracle, n, restart, steps):
    from warp_preconditioners_gb300 import linear

    if n == 40:
        steps = min(steps, 30)
    rng = np.random.default_rng(n)
    a = (ss.diags(2.3 + rng.uniform(0, 0.2, n)) + ss.diags(np.full(n - 1, -1.2), -1)
         + ss.diags(np.full(n - 1, -0.9), 1)).tocsr()
    b_np = rng.normal(size=n)
    xs = []
    for use_graph in (True, False):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        nit, res, _ = linear.gmres(to_bsr(a), vec(b_np), x, tol=0.0, restart=restart,
                                   maxiter=steps, use_cuda_graph=use_graph)
        xs.append(x.cpu().numpy())
    xo, ito, reso, _ = oracle.gmres(oracle.Operator.csr(oracle_csr(oracle, a)), b_np, tol=0.0,
                                    restart=restart, maxiter=steps)
    assert nit == ito == steps
    np.testing.assert_array_equal(xs[0], xs[1])
    # Twice-applied Gram-Schmidt keeps the basis orthogonal to rounding; the
    # matrix's condition (below 50) bounds what the sums' order can change.
    np.testing.assert_allclose(xs[0], xo, rtol=0, atol=1e-11 * np.abs(xo).max())
    np.testing.assert_allclose(res, reso, rtol=1e-9, atol=1e-13 * np.linalg.norm(b_np))
