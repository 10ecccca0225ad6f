"""The factor launch of the FSAI build, with and without loads ahead, at row
counts on both sides of the line between them and at supports on both sides of
its batches of 8, bit for bit against the oracle."""

import numpy as np
import pytest

from gpu_helpers import host_csr, oracle_csr, to_bsr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,width,step", [
    (161, 48, 2), (162, 48, 1),  # a third of a full GPU's threads at width 48: 25,941 rows
    (241, 8, 1), (242, 8, 3),    # and at width 8: 58,368
    (20, 7, 1), (20, 8, 2), (20, 9, 1), (20, 10, 3), (20, 16, 2), (20, 17, 1), (20, 25, 4),
    (20, 64, 1), (1, 8, 1)])
def test_factor_launch(oracle, side, width, step):
    import scipy.sparse as ss

    from warp_preconditioners_gb300 import FSAI, problems

    a = problems.laplacian_2d(side) if side > 1 else ss.csr_matrix([[3.0]])
    pre = FSAI(to_bsr(a), max_row_size=width, max_step_size=step, kap_tolerance=0.0)
    g, gt, _ = oracle.fsai(oracle_csr(oracle, a), width=width, step=step, tol=0.0)
    for m, o in ((pre.G, g), (pre.GT, gt)):
        off, col, val = host_csr(m)
        np.testing.assert_array_equal(off, o.offsets)
        np.testing.assert_array_equal(col, o.columns)
        np.testing.assert_array_equal(val, o.values)
