"""The factor applied to two interleaved vectors gives the bits of the product
with the 2 x 2 blocks g I_2, non-finite components included."""

import numpy as np
import pytest
import torch

from gpu_helpers import cuda, to_bsr

pytestmark = pytest.mark.gpu

STORES = [{}, {"factor_dtype": torch.float32}]


def pair_and_blocks(side, width, store):
    """RepeatedFSAI, and one whose operator holds the 2 x 2 blocks."""
    import scipy.sparse as ss

    from warp_preconditioners_gb300 import FSAI, RepeatedFSAI, _lib, problems

    a = problems.laplacian_2d(side) if side > 1 else ss.csr_matrix([[3.0]])
    factor = FSAI(to_bsr(a), max_row_size=width, **store)
    pair, blocks = RepeatedFSAI(factor), RepeatedFSAI(factor)
    blocks._op = _lib.new_op(
        "gbpc_op_fsai", a.shape[0], 2, _lib.ptr(blocks.G.offsets), _lib.ptr(blocks.G.columns),
        _lib.ptr(blocks.G.values), _lib.ptr(blocks.GT.offsets), _lib.ptr(blocks.GT.columns),
        _lib.ptr(blocks.GT.values), _lib.dtype_code(blocks.G.scalar_type),
        _lib.dtype_code(factor.dtype), _lib.stream(cuda()))
    return a, pair, blocks


@pytest.mark.parametrize("store", STORES)
@pytest.mark.parametrize("side,width", [(1, 4), (5, 8), (6, 1), (33, 5), (90, 48), (420, 8)])
def test_same_bits_as_blocks(side, width, store):
    a, pair, blocks = pair_and_blocks(side, width, store)
    n = a.shape[0]
    rng = np.random.default_rng(side)
    buf = torch.as_tensor(rng.normal(size=2 * n + 1), device=cuda()).to(pair.dtype)
    y = torch.as_tensor(rng.normal(size=2 * n), device=cuda()).to(pair.dtype)
    for x in (buf[:2 * n], buf[1:]):  # aligned for one load of both components, and not
        for alpha, beta in ((1.0, 0.0), (0.75, -1.5), (0.0, 2.0)):
            z1, z2 = torch.empty_like(y), torch.empty_like(y)
            pair.matvec(x, y, z1, alpha, beta)
            blocks.matvec(x, y, z2, alpha, beta)
            assert torch.equal(z1, z2), (alpha, beta)
    x = buf[:2 * n].clone()
    pair.matvec(buf[:2 * n], z1, z1, 1.0, 0.0)
    pair.matvec(x, x, x, 1.0, 0.0)  # all three the same vector
    assert torch.equal(x, z1)


def test_bfloat16_factors_stay_refused():
    with pytest.raises(ValueError, match="float64 or float32"):
        pair_and_blocks(5, 8, {"factor_dtype": torch.bfloat16})


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1.7e308])
def test_non_finite_components(bad):
    a, pair, blocks = pair_and_blocks(33, 8, {})
    n = a.shape[0]
    for where in (0, 7, 2 * n - 1):
        x = torch.as_tensor(np.random.default_rng(1).normal(size=2 * n), device=cuda())
        x[where] = bad
        z1, z2 = torch.empty_like(x), torch.empty_like(x)
        pair.matvec(x, z1, z1, 1.0, 0.0)
        blocks.matvec(x, z2, z2, 1.0, 0.0)
        np.testing.assert_array_equal(z1.cpu().numpy(), z2.cpu().numpy())


@pytest.mark.parametrize("side", [12, 70])
def test_fused_dot_in_cg(side):
    """CG on kron(A, I_2): the same iterates with either operator."""
    import scipy.sparse as ss

    from warp_preconditioners_gb300 import linear

    a, pair, blocks = pair_and_blocks(side, 8, {})
    A = to_bsr(ss.kron(a, ss.eye(2)).tocsr())
    b = torch.as_tensor(np.random.default_rng(3).normal(size=2 * a.shape[0]), device=cuda())
    xs = []
    for M in (pair, blocks):
        x = torch.zeros_like(b)
        linear.cg(A, b, x, tol=0.0, maxiter=20, M=M, check_every=0)
        xs.append(x)
    assert torch.equal(xs[0], xs[1])
