"""Row indices outside an LP's rows are refused by every host entry point, before an iteration runs."""
import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W
from vajra_pdhg.autograd import unrolled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index", [-1, 60, 2**31 - 1])
@pytest.mark.parametrize("where", [0, 1])
def test_row_index_out_of_range_is_refused(cuda, where, index):
    lps = [W.random_planted(60, 150, 4, seed=q) for q in range(2)]
    good = V.solve_batch(lps)
    lps[where].row_idx = lps[where].row_idx.copy()
    lps[where].row_idx[17] = index
    with pytest.raises(RuntimeError, match="row index out of range"):
        V.solve(lps[where])
    with pytest.raises(RuntimeError, match="row index out of range"):
        V.solve_batch(lps)
    with pytest.raises(RuntimeError, match="invalid argument"):
        unrolled(lps, np.ones(300), iterations=8)
    lps[where] = W.random_planted(60, 150, 4, seed=where)
    for a, b in zip(V.solve_batch(lps), good):   # and the library goes on
        np.testing.assert_array_equal(a["x"], b["x"])
