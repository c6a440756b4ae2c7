"""Sliced ELL over windows of 256 rows (the packed SpMVs of a batch), forced by shape -3."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu


def with_long_rows(lp, rows, cols, seed):
    """Rows and columns filled up to the given numbers of entries."""
    rng = np.random.default_rng(seed)
    a = lp.to_scipy_csc().tolil()
    for r, k in rows.items():
        a[r, rng.permutation(lp.num_cols)[:k]] = rng.uniform(0.1, 1.0, k)
    for c, k in cols.items():
        a[rng.permutation(lp.num_rows)[:k], c] = rng.uniform(0.1, 1.0, k)[:, None]
    a[[2, 3], :] = 0
    a[:, [5, lp.num_cols - 1]] = 0
    a = a.tocsc()
    a.eliminate_zeros()
    a.sort_indices()
    lp.col_ptr, lp.row_idx, lp.values = a.indptr.astype(np.int64), a.indices.astype(np.int32), a.data
    lp.row_lower = np.where(np.isin(np.arange(lp.num_rows), [2, 3]), -1.0, lp.row_lower)
    lp.row_upper = np.where(np.isin(np.arange(lp.num_rows), [2, 3]), 1.0, lp.row_upper)
    return lp


def batch(kind):
    if kind == "windows":      # one row past a window, a window exactly, one short of it, one row
        return [W.random_planted(m, n, (1, 9), seed=m) for m, n in ((257, 513), (256, 512), (255, 511), (1, 1), (2, 3))]
    if kind == "long":         # empty rows and columns; rows at 127, 128, 129 entries and above 4,096
        return [with_long_rows(W.random_planted(600, 6000, 3, seed=1), {0: 127, 300: 128, 301: 129, 599: 4097}, {7: 300, 5000: 128}, 2),
                W.random_planted(300, 700, (2, 40), seed=3)]
    return [W.random_planted(4001, 9003, (4, 12), seed=4), W.random_planted(37, 90, 3, seed=5), W.random_planted(999, 2500, 8, seed=6)]


@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
@pytest.mark.parametrize("kind", ["windows", "long", "uneven"])
def test_windows_match_the_lane_groups(cuda, kind, prec):
    """64 iterations against the set-up heuristic's lane groups: only the order of the row sums
    differs, so a sum of at most 4,097 products errs by 4,097 eps of its size and the iterates,
    through 64 nonexpansive steps, by at most 128 times that; a misplaced entry differs at O(1)."""
    lps = batch(kind)
    kw = dict(precision=prec, iteration_limit=64, tolerance=1e-30, autotune=0)
    eps = 2.0 ** -53 if prec == V.PREC_FP64 else 2.0 ** -24
    for a, b in zip(V.solve_batch(lps, spmv_shape_a=-3, spmv_shape_at=-3, **kw), V.solve_batch(lps, spmv_shape_a=1, **kw)):
        assert a["spmv_group_a"] == a["spmv_group_at"] == 130
        assert a["iterations"] == b["iterations"] == 64
        for k in ("x", "y", "row_value", "d"):
            np.testing.assert_allclose(a[k], b[k], rtol=0, atol=128 * 4097 * eps * (1e-3 + np.abs(b[k]).max()), err_msg=k)


def test_windows_reach_the_optima_as_instances_finish(cuda):
    """List mode: windows of finished instances are left out."""
    lps = batch("uneven") + [W.random_planted(m, 2 * m + 11, (3, 9), seed=m) for m in (64, 300, 700, 2200)]
    for lp, r in zip(lps, V.solve_batch(lps, spmv_shape_a=-3, spmv_shape_at=-3, tolerance=1e-5)):
        assert r["status_name"] == "OPTIMAL", r["status_message"]
        assert abs(r["objective_value"] - lp.planted_objective) <= 1e-3 * (1 + abs(lp.planted_objective))
