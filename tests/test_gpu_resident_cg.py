"""Cluster CG with the system in shared memory: sizes around slices and CTAs,
against the oracle, and bit-equal in groups where it runs from global memory."""

import numpy as np
import pytest
import scipy.sparse as ss
import torch

from gpu_helpers import cuda, oracle_csr, to_bsr, vec

pytestmark = pytest.mark.gpu


def _spd(n, seed):
    """A ragged pattern (rows sorted by length inside windows) with a dominant diagonal."""
    rng = np.random.default_rng(seed)
    a = ss.random(n, n, density=min(1.0, 5.0 / n), random_state=rng, format="csr")
    a = a + a.T
    return ss.csr_matrix(a + ss.diags(1.1 * np.asarray(abs(a).sum(axis=1)).ravel() + 0.1))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 511, 513, 1000, 4097])
@pytest.mark.parametrize("precond", [True, False])
def test_sizes_against_oracle(oracle, n, precond):
    from warp_preconditioners_gb300 import FSAI, linear

    a = _spd(n, n)
    b = np.random.default_rng(n).normal(size=n)
    A = to_bsr(a)
    M = FSAI(A, max_row_size=6) if precond else None
    x = torch.zeros(n, dtype=torch.float64, device=cuda())
    s = linear.Solver("cg", A, M)
    assert s.cluster_size > 0
    hist = torch.zeros(n + 2, dtype=torch.float64, device=cuda())
    nit, rr, _ = s.run(vec(b), x, tol=1e-10, history=hist)
    k = int(nit.item())
    h = hist.cpu().numpy()
    assert np.isclose(h[k] ** 2, float(rr.item()), rtol=1e-12)
    assert h[k] <= 1e-10 * np.linalg.norm(b) or k == n
    A_or = oracle.Operator.csr(oracle_csr(oracle, a))
    M_or = None
    if precond:
        g, gt, _ = oracle.fsai(oracle_csr(oracle, a), width=6)
        M_or = oracle.Operator.fsai(g, gt)
    x_or, it_or = oracle.krylov("cg", A_or, b, M=M_or, tol=1e-10)[:2]
    assert abs(k - it_or) <= 1
    if k < n:
        # Both residuals are at most 1e-10 |b| (and rounding far below that).
        d = a @ (x.cpu().numpy() - x_or)
        assert np.linalg.norm(d) <= 2.01e-10 * np.linalg.norm(b)
    # The same with a graph of separate kernels.
    y = torch.zeros_like(x)
    s2 = linear.Solver("cg", A, M, use_cuda_graph=False)
    nit2, _, _ = s2.run(vec(b), y, tol=1e-10)
    assert abs(int(nit2.item()) - k) <= 1


def test_groups_give_the_same_bits():
    """Alone (shared memory), in a small group, and in one too large for it."""
    from warp_preconditioners_gb300 import FSAI, linear
    from warp_preconditioners_gb300.multi import ClusterSolver

    sizes = [40, 700, 5000, 6000] + [900 + 17 * i for i in range(12)]
    systems, bs, alone = [], [], []
    for i, n in enumerate(sizes):
        A = to_bsr(_spd(n, i))
        M = FSAI(A, max_row_size=8)
        b = vec(np.random.default_rng(i).normal(size=n))
        x = torch.zeros_like(b)
        linear.Solver("cg", A, M).run(b, x, tol=1e-9)
        systems.append((A, M))
        bs.append(b)
        alone.append(x)
    for count in (3, len(sizes)):
        xs = [torch.zeros_like(b) for b in bs[:count]]
        ClusterSolver(systems[:count]).run(bs[:count], xs, tol=1e-9)
        assert all(torch.equal(p, q) for p, q in zip(xs, alone))
