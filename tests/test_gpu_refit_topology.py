"""The refit's own topology comparison: what it must refuse, at the ends of the
arrays and at unaligned storage, and what it leaves untouched."""

import numpy as np
import pytest
import scipy.sparse as ss
import torch

from gpu_helpers import cuda, host_csr, oracle_csr, to_bsr

pytestmark = pytest.mark.gpu


def _matrix(n=401):
    from warp_preconditioners_gb300 import problems

    return ss.csr_matrix(problems.laplacian_1d(n) + 0.01 * ss.eye(n))


def _fresh(a):
    from warp_preconditioners_gb300 import FSAI

    return FSAI(to_bsr(a), max_row_size=6, kap_tolerance=0.0, reuse_pattern=True)


@pytest.mark.parametrize("where", ["offset", "first", "last", "before_tail"])
@pytest.mark.parametrize("shift", [0, 1])
def test_differences_refused_factor_kept(oracle, where, shift):
    from warp_preconditioners_gb300.sparse import BsrMatrix

    a = _matrix()
    pre = _fresh(a)
    before = pre.G.values.clone()
    m = to_bsr(a)
    off = m.offsets.clone()
    # Columns at an address that is not a multiple of 16 bytes for shift 1.
    room = torch.empty(m.nnz + shift, dtype=torch.int32, device=cuda())
    col = room[shift:]
    col.copy_(m.columns)
    if where == "offset":
        off[1:2] += 1
    elif where == "first":
        col[:1] += 1
    elif where == "last":
        col[-1:] -= 1
    else:
        col[m.nnz // 4 * 4 - 1] += 1
    with pytest.raises(ValueError, match="identical sparsity"):
        pre.update(BsrMatrix(m.nrow, m.ncol, (1, 1), off, col, m.values * 2.0))
    assert torch.equal(pre.G.values, before)
    # The same storage with the right topology is accepted.
    col.copy_(m.columns)
    pre.update(BsrMatrix(m.nrow, m.ncol, (1, 1), m.offsets, col, m.values * 4.0))
    goff, gcol, gval = host_csr(pre.G)
    want, _, bad = oracle.fsai_refit(oracle_csr(oracle, a * 4.0), oracle.CSR(goff, gcol, gval))
    assert bad == 0
    np.testing.assert_array_equal(gval, want)


@pytest.mark.parametrize("width", [1, 2, 7, 8, 9])
def test_row_refit_bit_exact(oracle, width):
    """Support sizes around the widths of the thread-per-row refit."""
    from warp_preconditioners_gb300 import FSAI

    rng = np.random.default_rng(width)
    n = 130
    a = ss.random(n, n, density=0.06, random_state=rng, format="csr")
    a = a + a.T + ss.diags(np.asarray(abs(a + a.T).sum(axis=1)).ravel() + 1.0)
    pre = FSAI(to_bsr(a), max_row_size=width, kap_tolerance=0.0, reuse_pattern=True)
    off, col, val = host_csr(pre.G)
    new = ss.csr_matrix(a.multiply(1.0 + 0.05 * np.cos(np.arange(n))[:, None]
                                   * np.cos(np.arange(n))[None, :]))
    pre.update(to_bsr(new))
    want, _, bad = oracle.fsai_refit(oracle_csr(oracle, new), oracle.CSR(off, col, val))
    assert bad == 0
    np.testing.assert_array_equal(pre.G.values.cpu().numpy(), want)
