"""A wait between the CTAs of a cluster that runs out comes back as VAJRA_ERR_WAIT_TIMEOUT, on every path,
and leaves the context usable.  VAJRA_CLUSTER_WAIT_TRIES=0 (read once, hence a process of its own) makes every
thread give up on its first exchange, whose copies are on their way; the kernels end by themselves."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
sys.path[:0] = [%(root)r, %(root)r + "/vajra-opt_b200"]
import numpy as np
import vajra_pdhg as V
from vajra_pdhg import workloads as W
from vajra_pdhg.autograd import PREC_FP32, PREC_FP64, PREC_MIXED, unrolled

small, several = W.random_planted(60, 150, 4, seed=1), W.random_planted(2000, 5000, 8, seed=2)
fp32_only = W.random_planted(3000, 7000, 8, seed=3)          # FP64 does not fit: the norm is estimated packed
batch = [W.random_planted(1000, 2400, 8, seed=q) for q in range(3)]
ones = np.ones(sum(lp.num_cols for lp in batch))
calls = {
    "norm": lambda: V.solve(several, precision=V.PREC_FP64),
    "iterations": lambda: V.solve(fp32_only),
    "reference": lambda: V.solve(several, algorithm=V.ALGO_REFERENCE, iteration_limit=500),
    "batch64": lambda: V.solve_batch(batch, precision=V.PREC_FP64),
    "batch32": lambda: V.solve_batch(batch),
    "unrolled64": lambda: unrolled(batch, ones, iterations=1000, precision=PREC_FP64),
    "unrolled_mixed": lambda: unrolled(batch, ones, iterations=1000, precision=PREC_MIXED),
    "unrolled32": lambda: unrolled(batch, ones, iterations=1000, precision=PREC_FP32),
}
for _ in range(2):
    for name, call in calls.items():
        try:
            call()
        except RuntimeError as e:
            assert "timed out" in str(e), (name, e)
        else:
            sys.exit(name + ": no error")
        assert V.solve(small)["status_name"] == "OPTIMAL", name          # one CTA: nothing to wait for
large = W.random_planted(9000, 20000, 4, seed=5)                         # no cluster holds it: two launches an iteration
r = V.solve(large)
assert r["status_name"] == "OPTIMAL" and abs(r["objective_value"] - large.planted_objective) < 1e-3 * abs(large.planted_objective)
print("ok")
"""


def test_a_wait_that_runs_out_is_an_error_and_no_more(cuda):
    r = subprocess.run([sys.executable, "-c", CHILD % dict(root=ROOT)], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "VAJRA_CLUSTER_WAIT_TRIES": "0"})
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:] + r.stderr[-2000:]
