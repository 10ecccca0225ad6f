"""FSAI setup kernels at the sizes and patterns where their work split can go
wrong, bit for bit against the oracle."""

import numpy as np
import pytest
import scipy.sparse as ss

from gpu_helpers import host_csr, oracle_csr, to_bsr

pytestmark = pytest.mark.gpu


def _spd(kind, n, seed=0):
    """Diagonally dominant symmetric patterns with scaled diagonals."""
    rng = np.random.default_rng(seed)
    if kind == "random":  # ragged rows, the mirrored entry rarely at the mirrored place
        a = ss.random(n, n, density=min(1.0, 9.0 / n), random_state=rng, format="lil")
    elif kind == "arrow":  # one long row and column among short ones
        a = ss.lil_matrix((n, n))
        a[n // 2, :] = rng.normal(size=n)
    else:  # band
        k = min(n - 1, 20)
        a = ss.diags([rng.normal(size=n - d) for d in range(k + 1)], range(k + 1), format="lil")
    a = ss.csr_matrix(a)
    a = a + a.T
    a.setdiag(0)
    a.eliminate_zeros()
    a = a + ss.diags(np.asarray(abs(a).sum(axis=1)).ravel() + 1.0)
    d = ss.diags(np.exp2(rng.integers(-20, 20, size=n)))
    return ss.csr_matrix(d @ a @ d)


def _same(pre, g, gt):
    for m, o in ((pre.G, g), (pre.GT, gt)):
        off, col, val = host_csr(m)
        np.testing.assert_array_equal(off, o.offsets)
        np.testing.assert_array_equal(col, o.columns)
        np.testing.assert_array_equal(val, o.values)


@pytest.mark.parametrize("kind", ["random", "arrow", "band"])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 257])
def test_equilibration_row_blocks(oracle, kind, n):
    from warp_preconditioners_gb300 import FSAI

    a = _spd(kind, n)
    pre = FSAI(to_bsr(a), max_row_size=8, kap_tolerance=0.0)
    g, gt, _ = oracle.fsai(oracle_csr(oracle, a), width=8, tol=0.0)
    _same(pre, g, gt)


def test_missing_transpose_is_refused():
    from warp_preconditioners_gb300 import FSAI

    for n, r, c in ((9, 8, 0), (40, 3, 30)):
        a = ss.lil_matrix(_spd("band", n))
        a[r, c] = 0.01  # outside the band or inside it, one side only
        a[c, r] = 0.0
        a = ss.csr_matrix(a)
        a.eliminate_zeros()
        with pytest.raises(Exception, match="structurally symmetric"):
            FSAI(to_bsr(a), max_row_size=4)


@pytest.mark.parametrize("width", [3, 8, 9, 16, 17, 33])
def test_finish_groups(oracle, width):
    """Lane groups of the finishing kernel: 8, 16, 32 lanes and two positions a lane."""
    from warp_preconditioners_gb300 import FSAI

    a = _spd("band", 67, seed=width)
    pre = FSAI(to_bsr(a), max_row_size=width, kap_tolerance=0.0)
    g, gt, _ = oracle.fsai(oracle_csr(oracle, a), width=width, tol=0.0)
    _same(pre, g, gt)


@pytest.mark.parametrize("longest", [63, 64, 65, 255, 256, 257, 1100])
@pytest.mark.parametrize("short", [1, 20])
def test_transpose_row_lengths(longest, short):
    """Transposed rows at the edges of the sorted lengths (narrow and wide
    averages, and rows left to the insertion sort)."""
    from warp_preconditioners_gb300.sparse import bsr_transposed

    n = 2000
    rng = np.random.default_rng(longest + short)
    a = ss.lil_matrix((n, n))
    for k in range(short):
        a.setdiag(rng.normal(size=n - 7 * k), 7 * k)
    a[rng.permutation(n)[:longest], 5] = 1.5
    a = ss.csr_matrix(a)
    a.eliminate_zeros()
    off, col, val = host_csr(bsr_transposed(to_bsr(a)))
    t = ss.csr_matrix(a.T)
    t.sort_indices()
    np.testing.assert_array_equal(off, t.indptr)
    np.testing.assert_array_equal(col, t.indices)
    np.testing.assert_array_equal(val, t.data)


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 1025, 33000])
@pytest.mark.parametrize("widest", [3, 1030])
def test_sliced_layout_and_schedule(n, widest):
    """Products over layouts with one slice, a partial last window, several
    slices per warp of the scheduling kernel, and slices too wide for it."""
    import torch
    from gpu_helpers import vec
    from warp_preconditioners_gb300.fsai import _product_op

    rng = np.random.default_rng(n + widest)
    m = max(n, widest)
    a = ss.random(n, m, density=min(1.0, 3.0 / m), random_state=rng, format="csr")
    row = ss.csr_matrix((np.ones(widest), (np.full(widest, n // 2), np.arange(widest))),
                        shape=(n, m))
    a = ss.csr_matrix(a + row)
    x = rng.normal(size=m)
    z = torch.empty(n, dtype=torch.float64, device="cuda")
    _product_op(to_bsr(a), torch.float64).apply(vec(x), None, z, 1.0, 0.0, z.device)
    ref = a @ x
    # Sums of up to `widest` products in another order than SciPy's.
    bound = (widest + 8) * 2.0 ** -52 * (abs(a) @ np.abs(x)) + 1e-300
    assert np.all(np.abs(z.cpu().numpy() - ref) <= bound)
