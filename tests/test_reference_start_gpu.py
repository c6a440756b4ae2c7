"""VAJRA_ALGO_REFERENCE from start points away from zero: x and x_bar start at 0 clamped to the
column bounds (pdhg.cpp:167-175), so the first dual step already depends on the bounds."""
import numpy as np
import pytest

import vajra_pdhg as V
from oracle import bindings as B
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu
INF = 1e20
BOUNDS = {"above": (1.0, 5.0), "below": (-5.0, -1.0), "fixed": (2.5, 2.5), "from": (3.0, INF), "up_to": (-INF, -2.0)}


def lp_of(kind, m, n, k):
    lp = W.random_planted(m, n, k, seed=m + n)
    kinds = list(BOUNDS) if kind == "all" else [kind]
    which = np.random.default_rng(n).integers(0, len(kinds) + 1, n)   # the last part keeps [0, 10]
    for q, name in enumerate(kinds):
        lp.col_lower[which == q], lp.col_upper[which == q] = BOUNDS[name]
    return lp


# one CTA, several CTAs, the widest cluster, and too many columns for a cluster
SIZES = [(20, 50, 3), (301, 807, 3), (2000, 5000, 8), (3300, 9000, 3)]


@pytest.mark.parametrize("scale", [True, False])
@pytest.mark.parametrize("limit", [1, 130])
@pytest.mark.parametrize("kind", ["all", *BOUNDS])
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_starts_clamped_to_the_bounds_equal_the_oracle(cuda, size, kind, limit, scale):
    lp = lp_of(kind, *size)
    kw = dict(iteration_limit=limit, check_frequency=50, tolerance=1e-9, gap_tolerance=1e-9)
    g = V.solve(lp, algorithm=V.ALGO_REFERENCE, enable_scaling=int(scale), **kw)
    o = B.port_solve(lp, enable_scaling=scale, **kw)
    for k in ("x", "y", "d", "row_value"):
        np.testing.assert_array_equal(g[k], o[k], err_msg=k)
    for k in ("status", "iterations", "objective_value", "restart_count", "primal_residual", "dual_residual"):
        assert g[k] == o[k], k
