"""Columns of equal counts numbered by their first row (degree ordering of FP64 solves)."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu


def flow(m, n):
    return W.min_cost_flow(m, n, seed=m + n)


def dense_columns(m, n):
    """Columns of 0, 1 and all m entries beside a flow's two: the counts' and the rows' key bits meet."""
    rng = np.random.default_rng(m)
    lp = W.min_cost_flow(m, n, seed=7)
    a = lp.to_scipy_csc().tolil()
    a[:, n // 2] = rng.standard_normal((m, 1))
    a[:, 0] = 0.0
    a[1:, n - 1] = 0.0
    a[0, n - 1] = 1.5
    csc = a.tocsc()
    csc.sort_indices()
    q = W.LP(**{**lp.__dict__})
    q.col_ptr, q.row_idx, q.values = csc.indptr.astype(np.int64), csc.indices.astype(np.int32), csc.data.copy()
    return q


@pytest.mark.parametrize("lp", [flow(2, 40), flow(127, 900), flow(128, 901), flow(129, 33), dense_columns(63, 300),
                                dense_columns(64, 257), dense_columns(255, 1025)], ids=lambda lp: f"{lp.num_rows}x{lp.num_cols}")
def test_numbering_by_first_row_gives_the_callers_results(cuda, lp):
    """64 FP64 iterations with and without the ordering differ by summation order only: at most
    64 iterations x ~2,000 additions x 1.1e-16, times the iterates' growth of one rounding (below 100),
    is 2e-9 of the largest entry; a wrong number would show at O(1)."""
    kw = dict(precision=V.PREC_FP64, iteration_limit=64, spmv_shape_a=-1, spmv_shape_at=-1)
    a = V.solve(lp, degree_order=1, **kw)
    b = V.solve(lp, degree_order=-1, **kw)
    assert a["iterations"] == b["iterations"]
    for k in ("x", "y", "d", "row_value"):
        np.testing.assert_allclose(a[k], b[k], rtol=0, atol=2e-9 * (1.0 + np.abs(b[k]).max()), err_msg=k)
