"""Which batches run on clusters: few or small instances, not those that take the clusters many rounds."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu


def launches(lps, prec, **kw):
    a, b = (V.solve_batch(lps, precision=prec, iteration_limit=n, tolerance=1e-30, mixed_switch_tolerance=1e-30,
                          mixed_stall_checks=0, **kw)[0]["kernel_launches"] for n in (64, 192))
    return b - a   # of two more chunks: 2 x 128 and more packed, none on clusters


@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
def test_small_batches_run_on_clusters_large_ones_packed(cuda, prec):
    small = [W.random_planted(200, 500, 8, seed=q) for q in range(4)]
    large = [W.random_planted(2000, 5000, 8, seed=q) for q in range(4)]
    for lps, on_clusters in ((small * 8, True), (small * 128, True), (large, True), (large * 16, False)):
        n = launches(lps, prec, autotune=0)
        assert n < 16 if on_clusters else n >= 256, (len(lps), lps[0].num_rows, n)
    # packed or not, the iterates of the first chunk are the same bits
    for a, b in zip(V.solve_batch(large * 16, precision=prec, iteration_limit=64, tolerance=1e-30, autotune=0),
                    V.solve_batch(large, precision=prec, iteration_limit=64, tolerance=1e-30, autotune=0)):
        np.testing.assert_array_equal(a["x"], b["x"])
        np.testing.assert_array_equal(a["y"], b["y"])


@pytest.mark.parametrize("prec", ["fp64", "mixed", "fp32"])
def test_unrolled_steps_enough_for_clusters_match_the_packed_map(cuda, prec):
    """300 steps pay for the clusters' start; beside an LP of 7,000 x 20,000 all run packed.  300 nonexpansive
    steps and their reverse, sums of at most 64 products: 2 x 300 x 64 eps of the largest entry."""
    from vajra_pdhg.autograd import PREC_FP32, PREC_FP64, PREC_MIXED, unrolled
    p = {"fp64": PREC_FP64, "mixed": PREC_MIXED, "fp32": PREC_FP32}[prec]
    lps = [W.random_planted(m, n, 6, seed=90 + m) for m, n in ((60, 150), (301, 807), (1000, 3000))] * 6
    big = W.random_planted(7000, 20000, 6, seed=9)
    n, m = sum(lp.num_cols for lp in lps), sum(lp.num_rows for lp in lps)
    w = np.random.default_rng(3).standard_normal(n + big.num_cols)
    a = unrolled(lps, w[:n], iterations=300, checkpoint_every=64, precision=p, enable_scaling=0)
    b = unrolled(lps + [big], w, iterations=300, checkpoint_every=64, precision=p, enable_scaling=0)
    e32, e64 = 2.0 ** -24, 2.0 ** -53
    for key, size, eps in (("x", n, e32 if prec == "fp32" else e64), ("loss", len(lps), e32 if prec == "fp32" else e64),
                           ("grad_c", n, e64 if prec == "fp64" else e32), ("grad_row_lower", m, e64 if prec == "fp64" else e32),
                           ("grad_row_upper", m, e64 if prec == "fp64" else e32)):
        u, v = a[key], b[key][:size]
        np.testing.assert_allclose(u, v, rtol=0, atol=2 * 300 * 64 * eps * (1.0 + np.abs(v).max()), err_msg=key)
