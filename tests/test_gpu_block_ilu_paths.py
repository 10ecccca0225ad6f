"""BlockILU0 setup and apply where their launches change: sweep counts, block
sizes, scalings and aliases, against the oracle."""

import numpy as np
import pytest
import scipy.sparse as ss
import torch

from gpu_helpers import to_bsr, vec

pytestmark = pytest.mark.gpu


def _matrix(nb, block, seed):
    """Diagonally dominant blocks on a ragged symmetric pattern."""
    rng = np.random.default_rng(seed)
    p = ss.random(nb, nb, density=min(1.0, 4.0 / nb), random_state=rng, format="csr")
    p = ((p + p.T) != 0).astype(float).tolil()
    p.setdiag(1.0)
    a = ss.kron(ss.csr_matrix(p), np.ones((block, block)), format="csr")
    a.data = rng.uniform(-1.0, 1.0, size=a.nnz)
    a = a + ss.diags(2.0 * np.asarray(abs(a).sum(axis=1)).ravel())
    return ss.bsr_matrix(ss.csr_matrix(a), blocksize=(block, block))


@pytest.mark.parametrize("block", [1, 2, 3, 4])
@pytest.mark.parametrize("sweeps", [1, 2, 3, 4])
def test_apply_sweeps_scalings_and_aliases(oracle, block, sweeps):
    from warp_preconditioners_gb300 import BlockILU0

    a = _matrix(67, block, 10 * block + sweeps)
    a.sort_indices()
    n = a.shape[0]
    pre = BlockILU0(to_bsr(a, block=block), factor_sweeps=2, solve_sweeps=sweeps)
    fac, inv = pre.factors.cpu().numpy(), pre.inverse_diagonal.cpu().numpy()
    rng = np.random.default_rng(sweeps)
    for alpha, beta in ((1.0, 0.0), (0.7, -0.3), (1.0, 0.5), (0.0, 2.0)):
        for alias in ("none", "xz", "yz"):
            x, y = rng.normal(size=n), rng.normal(size=n)
            ref = oracle.bilu0_apply(67, block, a.indptr, a.indices, fac, inv, sweeps, x, y,
                                     alpha, beta)
            xd, yd = vec(x), vec(y)
            zd = xd if alias == "xz" else yd if alias == "yz" else torch.empty_like(xd)
            pre.matvec(xd, yd, zd, alpha, beta)
            # A few hundred rounded operations a row on O(1) values.
            np.testing.assert_allclose(zd.cpu().numpy(), ref, rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("block", [1, 2, 3, 4])
@pytest.mark.parametrize("relaxation", [1.0, 0.8])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_factor_sweeps_bit_exact(oracle, block, relaxation, dtype):
    from warp_preconditioners_gb300 import BlockILU0

    a = _matrix(131, block, block)
    a.sort_indices()
    npdt = np.float64 if dtype == torch.float64 else np.float32
    pre = BlockILU0(to_bsr(a, dtype, block=block), factor_sweeps=3, solve_sweeps=2,
                    relaxation=relaxation)
    fac, inv = oracle.bilu0_setup(131, block, a.indptr, a.indices, a.data.astype(npdt),
                                  factor_sweeps=3, relaxation=relaxation)[:2]
    bits = np.int64 if dtype == torch.float64 else np.int32
    for got, want in ((pre.factors, fac), (pre.inverse_diagonal, inv)):
        np.testing.assert_array_equal(got.cpu().numpy().reshape(-1).view(bits),
                                      np.asarray(want, npdt).reshape(-1).view(bits))
