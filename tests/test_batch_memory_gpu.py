"""The batch's optional copies of the matrices over windows of 256 rows do not narrow what fits."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
sys.path[:0] = [%(root)r, %(root)r + "/vajra-opt_b200"]
import numpy as np, torch
import vajra_pdhg as V
from vajra_pdhg import workloads as W

lps = [W.random_planted(9000, 20000, 12, seed=q) for q in range(8)]
assert sum(lp.nnz for lp in lps) > 1 << 20          # windows are among the autotuner's shapes
kw = dict(precision=V.PREC_FP64, iteration_limit=64, tolerance=1e-30)

def call(autotune):
    try:
        return V.solve_batch(lps, autotune=autotune, **kw)
    except Exception as e:
        assert "memory" in str(e).lower(), e
        return None

want = call(1), call(0)                              # (loads the kernels)
torch.cuda.init()
step, rooms = 8 << 20, 0
for room in range(96 << 20, 1 << 30, step):
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    plain = call(0)
    if plain is not None:
        rooms += 1
        tuned = call(1)
        assert tuned is not None, (room, rooms)
        for a, b in zip(tuned, want[1]):
            for k in ("x", "y"):                     # other shapes add a row in another order: 64 steps x 40 products
                np.testing.assert_allclose(a[k], b[k], rtol=0, atol=64 * 40 * 1e-13 * (1 + np.abs(b[k]).max()))
    del hog
    torch.cuda.empty_cache()
    if rooms == 6:
        print("ok", room)
        sys.exit(0)
sys.exit("no room was enough")
"""


def test_a_batch_that_fits_without_windows_runs(cuda):
    """With ever more room, from the first that holds the call without the autotuner (no windows) on."""
    r = subprocess.run([sys.executable, "-c", CHILD % dict(root=ROOT)], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "VAJRA_BLOCK_CACHE_MB": "0"})
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
