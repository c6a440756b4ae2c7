"""Hand-over from an FP32 phase on a thread-block cluster to an FP64 phase that does not fit one."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("switch", [1e3, 1e-3])
@pytest.mark.parametrize("mode", [0, 1])
def test_packed_fp64_phase_goes_on_from_the_clusters_state(cuda, mode, switch):
    """3,000 x 7,000, 8 entries a column: a cluster holds the FP32 copy, not the FP64 one.  The FP32
    phase ends at its first check, or a few checks later, and the FP64 phase runs one chunk, against the
    two-launch iteration in both phases.  A hand-over at the first check comes before any restart: the
    same bits.  After a restart the checks' FP64 sums, in another order, move the step sizes by one
    rounding of their FP32 copies at most, over the iterations run."""
    lp = W.random_planted(3000, 7000, 8, seed=31)
    kw = dict(handover_mode=mode, tolerance=1e-30, mixed_switch_tolerance=switch, spmv_shape_a=16, spmv_shape_at=4)
    fp32 = V.solve(lp, iteration_limit=4096, **kw)["fp32_iterations"]
    assert fp32 == 64 if switch > 1.0 else 64 < fp32 < 4096
    b = V.solve(lp, iteration_limit=fp32 + 64, **kw)
    a = V.solve(lp, iteration_limit=fp32 + 64, **{**kw, "spmv_shape_a": 0, "spmv_shape_at": 0})
    assert a["kernel_launches"] < b["kernel_launches"] - fp32          # the FP32 phase ran on a cluster
    assert a["kernel_launches"] >= 128                                 # the FP64 chunk did not
    assert (a["spmv_group_a"], a["spmv_group_at"]) == (16, 4)          # the same row sums
    for k in ("iterations", "fp32_iterations", "fp64_iterations", "restart_count"):
        assert a[k] == b[k], k
    assert a["fp64_iterations"] == 64
    for k in ("x", "y", "row_value", "d"):
        if switch > 1.0:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
        else:
            bound = a["iterations"] * 2.0 ** -24 * (1.0 + np.abs(b[k]).max())
            np.testing.assert_allclose(a[k], b[k], rtol=0, atol=bound, err_msg=k)
