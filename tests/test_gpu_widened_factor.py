"""Products with float32 and bfloat16 storage on float64 vectors: every stored
value is widened exactly."""

import numpy as np
import pytest
import scipy.sparse as ss
import torch

from gpu_helpers import cuda, to_bsr, vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["", "0", "3"])
@pytest.mark.parametrize("storage", [torch.float32, torch.bfloat16])
def test_stored_values_widened_exactly(monkeypatch, variant, storage):
    from warp_preconditioners_gb300 import _lib

    if variant:
        monkeypatch.setenv("GBPC_SPMV_VARIANT", variant)
    tiny = np.array([1.0e-45, 1.4e-42, 1.1754942e-38, 1.17549435e-38, 2.5e-38, 3.4028234e38,
                     1.0, -1.0, 0.0, -0.0, 1 / 3, 65504.0, -1.0e-40, np.inf, -np.inf, np.nan])
    rng = np.random.default_rng(0)
    stored = torch.as_tensor(np.concatenate([tiny, rng.normal(size=500) * np.exp2(
        rng.integers(-140, 120, size=500))]), dtype=torch.float32).to(storage)
    n = stored.numel()
    diag = ss.eye(n, format="csr")
    b = to_bsr(diag, torch.float32)
    b.values = stored.to(cuda())
    one = to_bsr(diag, torch.float32)
    one.values = torch.ones(n, dtype=storage, device=cuda())
    op = _lib.new_op("gbpc_op_fsai", n, 1, *[_lib.ptr(q) for q in (
        b.offsets, b.columns, b.values, one.offsets, one.columns, one.values)],
        _lib.dtype_code(storage), _lib.GBPC_F64, _lib.stream(cuda()))
    z = torch.empty(n, dtype=torch.float64, device=cuda())
    op.apply(vec(np.ones(n)), None, z, 1.0, 0.0, cuda())
    # 0 + v * 1, then 0 + 1 * that: the value itself (zeros lose their sign).
    np.testing.assert_array_equal(z.cpu().numpy(), stored.to(torch.float64).numpy())


@pytest.mark.parametrize("factor_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("side", [1, 5, 33, 90])
def test_float32_apply_writes_float64(factor_dtype, side):
    """The product that writes float64 itself gives the bits of the widening
    kernel (alpha = 1, beta = 1 with y = 0), eagerly and in a captured graph."""
    from warp_preconditioners_gb300 import FSAI, problems

    a = problems.laplacian_2d(side) if side > 1 else ss.csr_matrix([[3.0]])
    pre = FSAI(to_bsr(a), max_row_size=8, factor_dtype=factor_dtype, apply_dtype=torch.float32)
    n = a.shape[0]
    x = vec(np.random.default_rng(side).normal(size=n))
    zeros, z1, z2 = torch.zeros_like(x), torch.empty_like(x), torch.empty_like(x)
    pre.matvec(x, z1, z1, 1.0, 0.0)
    pre.matvec(x, zeros, z2, 1.0, 1.0)
    assert torch.equal(z1, z2)
    xz = x.clone()
    pre.matvec(xz, xz, xz, 1.0, 0.0)  # all three the same vector
    assert torch.equal(xz, z1)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        pre.matvec(x, z2, z2, 1.0, 0.0)
    z2.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(z1, z2)
