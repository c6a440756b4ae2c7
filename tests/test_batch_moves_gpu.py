"""Batches whose instances change path between two launches of a pass: packed to clusters, when the
instances too large for a cluster have finished, and the widths of clusters as instances finish."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "row_value", "d")
FIRST = 2048   # iterations of a pass's first launch


def solved_at_once(lp):
    """The same matrix with c = 0 and rows that hold at the start point: optimal at the first check."""
    lp.c = np.zeros(lp.num_cols)
    lp.row_lower, lp.row_upper = np.full(lp.num_rows, -1.0), np.full(lp.num_rows, 1.0)
    return lp


def options(prec, limit):
    kw = dict(precision=prec, iteration_limit=limit, tolerance=1e-30, autotune=0)
    if prec == V.PREC_MIXED:   # the FP32 pass goes on to the limit
        kw.update(mixed_switch_tolerance=1e-30, mixed_stall_checks=0)
    return kw


@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
def test_packed_instances_that_move_to_clusters_repeat_bit_for_bit(cuda, prec):
    """More than 4M entries outside clusters: all run packed.  Those finish at the first check, one
    of 9,000 x 20,000 stays packed, and from the second launch on the others run on clusters beside it."""
    lps = [solved_at_once(W.random_planted(5000, 21000, 210, seed=1)), W.random_planted(9000, 20000, 3, seed=2)]
    assert lps[0].nnz > 4 << 20
    lps += [W.random_planted(60 + 13 * q, 150 + 31 * q, (2, 7), seed=10 + q) for q in range(24)]
    kw = options(prec, FIRST + 1024)
    a, b = V.solve_batch(lps, **kw), V.solve_batch(lps, **kw)
    assert a[0]["iterations"] == 64
    for u, v in zip(a, b):
        assert u["iterations"] == v["iterations"] and u["restart_count"] == v["restart_count"]
        assert u["rel_kkt"] == v["rel_kkt"]
        for k in KEYS:
            np.testing.assert_array_equal(u[k], v[k], err_msg=k)
    # The packed iteration throughout (a fixed shape) has the same row sums; only the FP64 sums of the
    # checks are added in another order: 4 x 20,000 eps in the primal weight, so in the step sizes (or one rounding of
    # their FP32 copies), over 1,024 nonexpansive iterations.
    assert sum(r["restart_count"] for r in a[2:]) > 24
    bound = 1024 * (4 * 20000 * 2.0 ** -53 if prec == V.PREC_FP64 else 2.0 ** -24)
    for u, v in zip(a[1:], V.solve_batch(lps, spmv_shape_a=1, **kw)[1:]):
        assert u["iterations"] == v["iterations"] == FIRST + 1024 and u["restart_count"] == v["restart_count"]
        for k in KEYS:
            np.testing.assert_allclose(u[k], v[k], rtol=0, atol=bound * (1.0 + np.abs(v[k]).max()), err_msg=k)


def singletons_first(seed):
    """1,000 x 2,400: 300 columns of one entry, then 2,100 of 15.  Equal shares of the entries give a
    CTA of 8 (512 threads) up to 420 columns, one of 16 (256 threads) 260: the wider cluster does not
    hold it."""
    lp = W.random_planted(1000, 2400, 15, seed=seed)
    a = lp.to_scipy_csc().tolil()
    for j in range(300):
        a[:, j] = 0.0
        a[(7 * j) % 1000, j] = 1.0 + 0.01 * j
    a = a.tocsc()
    a.eliminate_zeros()
    a.sort_indices()
    x, y, z = lp.x_planted, lp.y_planted, lp.c - lp.to_scipy_csc().T @ lp.y_planted
    lp.col_ptr, lp.row_idx, lp.values = a.indptr.astype(np.int64), a.indices.astype(np.int32), a.data
    lp.row_lower = lp.row_upper = a @ x
    lp.c = a.T @ y + z
    return lp


@pytest.mark.parametrize("limit", [FIRST + 64, FIRST + 576])
@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
def test_an_instance_left_alone_goes_on_as_the_packed_iteration(cuda, prec, limit):
    """Nine of ten finish at the first check; for the second launch the tenth could have a cluster
    twice as wide, which does not hold it.  Bound as above, 2,624 iterations and 2,400 columns."""
    lps = [solved_at_once(singletons_first(q)) for q in range(9)] + [singletons_first(9)]
    kw = options(prec, limit)
    u, v = V.solve_batch(lps, **kw)[9], V.solve_batch(lps, spmv_shape_a=1, **kw)[9]
    assert u["iterations"] == v["iterations"] == limit and u["restart_count"] == v["restart_count"] > 0
    bound = 2624 * (4 * 2400 * 2.0 ** -53 if prec == V.PREC_FP64 else 2.0 ** -24)
    for k in KEYS:
        np.testing.assert_allclose(u[k], v[k], rtol=0, atol=bound * (1.0 + np.abs(v[k]).max()), err_msg=k)


@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
def test_a_cluster_that_holds_an_instance_is_kept(cuda, prec):
    """The same batch: the wider cluster's refusal costs the tenth LP nothing.  Sixteen more checks are
    sixteen packed chunks of 2 x 64 launches and more, or one launch of its cluster."""
    lps = [solved_at_once(singletons_first(q)) for q in range(9)] + [singletons_first(9)]
    a, b = (V.solve_batch(lps, **options(prec, FIRST + n)) for n in (64, 64 + 1024))
    assert a[9]["iterations"] == FIRST + 64 and b[9]["iterations"] == FIRST + 1088
    assert b[9]["kernel_launches"] - a[9]["kernel_launches"] < 128
