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
