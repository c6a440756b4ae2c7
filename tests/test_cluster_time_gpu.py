"""The time limit of an LP that runs on a thread-block cluster is looked at after its first check."""
import pytest

import vajra_pdhg as V
from vajra_pdhg import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [1, 64, 5000])
@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
@pytest.mark.parametrize("size", [(60, 150, 4), (500, 1200, 6), (9000, 20000, 3)], ids=str)   # one CTA, several, no cluster
def test_no_time_left_ends_after_the_first_check(cuda, size, prec, every):
    r = V.solve(W.random_planted(*size, seed=41), precision=prec, check_frequency=every, time_limit=0.0, tolerance=1e-30)
    assert r["status_name"] == "TIME_LIMIT" and r["iterations"] == every


@pytest.mark.parametrize("prec", [V.PREC_FP64, V.PREC_MIXED])
def test_a_generous_limit_changes_nothing(cuda, prec):
    lp = W.random_planted(500, 1200, 6, seed=42)
    a, b = V.solve(lp, precision=prec), V.solve(lp, precision=prec, time_limit=3600.0)
    assert a["status_name"] == b["status_name"] == "OPTIMAL" and a["iterations"] == b["iterations"]
    assert (a["x"] == b["x"]).all() and (a["y"] == b["y"]).all()
