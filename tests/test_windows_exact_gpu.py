"""Sliced ELL over windows adds a row's products in storage order, one fused multiply-add after another:
the bits of one lane per row, whatever the places of the rows in their windows."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu


def lp_with_lengths(m, n, lengths, seed, transposed=False):
    """`lengths[q]` entries in row 97 q (of the columns, where transposed), none or one in the others."""
    rng = np.random.default_rng(seed)
    lines, places = (n, m) if transposed else (m, n)
    counts = rng.integers(0, 2, lines)
    counts[97 * np.arange(len(lengths))] = lengths
    r = np.repeat(np.arange(lines), counts)
    c = np.concatenate([rng.permutation(places)[:k] for k in counts]).astype(np.int64)
    if transposed:
        r, c = c, r
    col_ptr, row_idx, values = W.canonical_csc(m, n, r, c, rng.uniform(0.1, 10.0, r.size) * rng.choice([-1.0, 1.0], r.size))
    lower = -rng.uniform(0.0, 1.0, m)
    return W.LP(m, n, col_ptr, row_idx, values, rng.standard_normal(n), np.zeros(n), rng.uniform(1.0, 5.0, n), lower, lower + 1.0)


@pytest.mark.parametrize("limit", [1, 2, 64])
@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
def test_windows_have_the_bits_of_one_lane_a_row(cuda, prec, limit):
    """Fewer than two entries a line on average, so the set-up heuristic gives a row one lane; lines of up to
    128 entries (the longest that windows keep) beside lines of none and one, across window borders."""
    lengths = [128, 127, 65, 64, 3, 2, 33, 128, 126, 31, 5, 16, 127, 2]
    lps = [lp_with_lengths(1500, 1400, lengths, 1), lp_with_lengths(1400, 1500, lengths, 2, transposed=True),
           lp_with_lengths(255, 300, [2], 3), lp_with_lengths(1, 2, [2], 4)]
    kw = dict(precision=prec, iteration_limit=limit, tolerance=1e-30, autotune=0)
    for a, b in zip(V.solve_batch(lps, spmv_shape_a=-3, spmv_shape_at=-3, **kw), V.solve_batch(lps, spmv_shape_a=1, **kw)):
        assert a["spmv_group_a"] == a["spmv_group_at"] == 130 and b["spmv_group_a"] == b["spmv_group_at"] == 1
        # the norm estimate's row sums (60 rounds over windows) are the same bits too, so the step sizes are
        assert a["spectral_norm_estimate"] == b["spectral_norm_estimate"]
        for k in ("x", "y", "row_value", "d"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
