"""Cluster-resident iterations (one LP in the shared memory of a thread-block cluster): the same
row sums in the same order as the two-launch kernels, so the first 64 iterations -- up to the
first check, whose FP64 sums are the only ones in another order -- give the same bits."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W
from vajra_pdhg.kkt import relative_kkt

pytestmark = pytest.mark.gpu


def lp_of(kind):
    if kind == "one_row":            # a 16-byte slice of y, most CTAs without rows
        return W.random_planted(1, 700, 1, seed=3)
    if kind == "few_rows":           # 3 rows over several CTAs: empty slices
        return W.random_planted(3, 1500, (1, 3), seed=4)
    if kind == "dense_row":          # a row of 1,999 entries (256 threads) beside rows of a few
        lp = W.random_planted(400, 2000, 3, seed=5)
        a = lp.to_scipy_csc().tolil()
        a[7, : 1999] = np.random.default_rng(1).uniform(0.5, 1.0, 1999)
        a = a.tocsc()
        a.sort_indices()
        lp.col_ptr, lp.row_idx, lp.values = a.indptr.astype(np.int64), a.indices.astype(np.int32), a.data
        return lp
    if kind == "empty":              # empty rows and columns
        lp = W.random_planted(300, 800, 2, seed=6)
        a = lp.to_scipy_csc().tolil()
        a[[0, 5, 299], :] = 0
        a[:, [0, 17, 799]] = 0
        a = a.tocsc()
        a.eliminate_zeros()
        a.sort_indices()
        lp.col_ptr, lp.row_idx, lp.values = a.indptr.astype(np.int64), a.indices.astype(np.int32), a.data
        lp.row_lower = np.where(np.isin(np.arange(300), [0, 5, 299]), -1.0, lp.row_lower)
        lp.row_upper = np.where(np.isin(np.arange(300), [0, 5, 299]), 1.0, lp.row_upper)
        return lp
    m, n, k = kind
    return W.random_planted(m, n, k, seed=m + n)


CASES = ["one_row", "few_rows", "dense_row", "empty", (2, 2, 1), (60, 150, 4), (255, 256, 3), (257, 257, 4),
         (301, 807, 3), (100, 400, 40), (1000, 1001, (1, 30)), (2000, 5000, 8), (2003, 5003, (4, 12)), (3000, 7001, 2)]


@pytest.mark.parametrize("limit", [1, 64])
@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
@pytest.mark.parametrize("kind", CASES, ids=str)
def test_same_bits_as_the_two_launch_iteration(cuda, kind, prec, limit):
    lp = lp_of(kind)
    kw = dict(precision=prec, iteration_limit=limit, tolerance=1e-30)
    a = V.solve(lp, **kw)
    b = V.solve(lp, spmv_shape_a=a["spmv_group_a"], spmv_shape_at=a["spmv_group_at"], **kw)   # forced shapes: two launches
    assert a["kernel_launches"] < b["kernel_launches"]   # one launch for the chunk
    assert a["iterations"] == b["iterations"] == limit
    for k in ("x", "y", "row_value", "d"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    # the check's FP64 sums: at most ~3 n additions in another order, n <= 7,001, then a square root
    assert abs(a["rel_kkt"] - b["rel_kkt"]) <= 4 * 7001 * 2.3e-16 * (1.0 + b["rel_kkt"])


@pytest.mark.parametrize("kw", [dict(check_frequency=7), dict(check_frequency=300), dict(restart_metric=1),
                                dict(max_violation=1e-5), dict(degree_order=1), dict(handover_mode=1)], ids=str)
def test_options_reach_the_optimum(cuda, kw):
    lp = W.random_planted(500, 1200, 6, seed=21)
    g = V.solve(lp, **kw)
    assert g["status_name"] == "OPTIMAL" and relative_kkt(lp, g["x"], g["y"])["rel_kkt"] <= 1.05e-6
    assert abs(g["objective_value"] - lp.planted_objective) <= 1e-5 * (1 + abs(lp.planted_objective))


def test_limit_in_the_middle_of_a_chunk_and_a_resident_rerun(cuda):
    lp = W.random_planted(500, 1200, 6, seed=22)
    with V.Solver(lp, precision=V.PREC_FP64, iteration_limit=150, tolerance=1e-30) as s:
        a, b = s.run(), s.run()
    assert a["iterations"] == b["iterations"] == 150 and a["status_name"] == "ITERATION_LIMIT"
    for k in ("x", "y", "row_value", "d"):
        np.testing.assert_array_equal(a[k], b[k])


BATCHES = {"tiny": [(2, 2, 1), (60, 150, 4), (255, 256, 3)],
           "spread": [(60, 150, 4), (301, 807, 3), (100, 400, 40), (1000, 1001, (1, 30)), (2000, 5000, 8), (4000, 9001, 6)],
           "odd": ["one_row", "few_rows", "dense_row", "empty", (61, 149, 3)],
           "one": [(500, 1200, 6)]}


@pytest.mark.parametrize("limit", [1, 64])
@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
@pytest.mark.parametrize("kind", sorted(BATCHES))
def test_batched_clusters_give_the_packed_iterations_bits(cuda, kind, prec, limit):
    """Instances on clusters (alone or beside instances that are too large for one) against the
    packed two-launch iteration (a fixed launch shape keeps the batch off the clusters)."""
    lps = [lp_of(k) for k in BATCHES[kind]]
    kw = dict(precision=prec, iteration_limit=limit, tolerance=1e-30, autotune=0)
    for a, b in zip(V.solve_batch(lps, **kw), V.solve_batch(lps, spmv_shape_a=1, **kw)):
        assert a["iterations"] == b["iterations"] == limit
        for k in ("x", "y", "row_value", "d"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
def test_batched_clusters_beside_larger_instances_reach_the_optima(cuda, prec):
    lps = [lp_of(k) for k in BATCHES["spread"] if k != (100, 400, 40)]
    for lp, r in zip(lps, V.solve_batch(lps, precision=prec, iteration_limit=40000)):
        assert r["status_name"] == "OPTIMAL" and relative_kkt(lp, r["x"], r["y"])["rel_kkt"] <= 1.05e-6
        assert r["fp32_iterations"] + r["fp64_iterations"] == r["iterations"]


@pytest.mark.parametrize("prec", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("every", [7, 100])
def test_unrolled_on_clusters_matches_the_packed_map(cuda, prec, every):
    """Alone, every instance fits a cluster; beside one of 7,000 x 20,000 all run packed.  Same row
    sums in the same order only where the packed matrices have the same mean row length, so the
    bound is rounding: 30 nonexpansive steps and their reverse, sums of at most 64 products, error
    <= 2 * 30 * 64 eps of the largest entry, eps the precision of the pass (the gradients of the
    mixed form come from FP32)."""
    from vajra_pdhg.autograd import PREC_FP32, PREC_FP64, PREC_MIXED, unrolled
    p = {"fp64": PREC_FP64, "mixed": PREC_MIXED, "fp32": PREC_FP32}[prec]
    lps = [W.random_planted(m, n, 6, seed=90 + m) for m, n in ((60, 150), (301, 807), (1000, 3000))]
    big = W.random_planted(7000, 20000, 6, seed=9)
    n = sum(lp.num_cols for lp in lps)
    m = sum(lp.num_rows for lp in lps)
    w = np.random.default_rng(3).standard_normal(n + big.num_cols)
    a = unrolled(lps, w[:n], iterations=30, checkpoint_every=every, precision=p, enable_scaling=0)
    b = unrolled(lps + [big], w, iterations=30, checkpoint_every=every, precision=p, enable_scaling=0)
    for key, size, eps in (("x", n, 2.0 ** -24 if prec == "fp32" else 2.0 ** -53),
                           ("loss", len(lps), 2.0 ** -24 if prec == "fp32" else 2.0 ** -53),
                           ("grad_c", n, 2.0 ** -53 if prec == "fp64" else 2.0 ** -24),
                           ("grad_row_lower", m, 2.0 ** -53 if prec == "fp64" else 2.0 ** -24),
                           ("grad_row_upper", m, 2.0 ** -53 if prec == "fp64" else 2.0 ** -24)):
        u, v = a[key], b[key][:size]
        np.testing.assert_allclose(u, v, rtol=0, atol=2 * 30 * 64 * eps * (1.0 + np.abs(v).max()), err_msg=key)


@pytest.mark.parametrize("kind", CASES + [(3300, 7400, 3)], ids=str)
def test_reference_algorithm_on_clusters_equals_the_oracle(cuda, kind):
    """The in-order row sums of the reference algorithm, bit for bit, at the edges of the slices and
    of the sums' tiles (1,024 terms)."""
    from oracle import bindings as B
    lp = lp_of(kind)
    kw = dict(iteration_limit=130, check_frequency=50, tolerance=1e-9, gap_tolerance=1e-9)
    g = V.solve(lp, algorithm=V.ALGO_REFERENCE, **kw)
    o = B.port_solve(lp, **kw)
    for k in ("x", "y", "d", "row_value"):
        np.testing.assert_array_equal(g[k], o[k], err_msg=k)
    assert g["status"] == o["status"] and g["iterations"] == o["iterations"] and g["objective_value"] == o["objective_value"]
