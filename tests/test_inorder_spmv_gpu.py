"""The in-order SpMV at the edges of its CTAs (1 to 256 rows), tiles (1,024 and 2,048 products) and of the
rows that a thread loads itself (up to 4 entries a row in CTAs of 256): products rounded, added in
storage order, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import vajra_pdhg as V
from vajra_pdhg import _capi, workloads as W

pytestmark = pytest.mark.gpu
FULL = 8 * 148 * 256   # rows from which a CTA takes 256 (on 148 SMs)


def lengths(kind):
    rng = np.random.default_rng(7)
    if isinstance(kind, int):                       # few rows, some far longer than a tile
        n = rng.integers(0, 40, kind)
        n[::max(1, kind // 5)] = [2047, 2048, 2049, 5000, 0, 1][: len(n[::max(1, kind // 5)])]
        return n
    n = np.full({"full": FULL, "full+1": FULL + 1, "full-1": FULL - 1}[kind], 4)
    n[256 * 3 + 17] = 5                             # 1,025 entries in a CTA
    n[256 * 5:256 * 6] = 0
    n[256 * 7:256 * 8] = 8                          # two tiles of 1,024
    n[256 * 9 + 255] = 3000
    n[256 * 11] = 1020 - 4 * 255 + 4                # 1,024 exactly
    n[-1] = 2051
    return n


def in_order(ptr, idx, val, x):
    s = np.zeros(ptr.size - 1, val.dtype)
    n = np.diff(ptr)
    order = np.argsort(-n, kind="stable")
    for k in range(int(n.max(initial=0))):
        r = order[: np.searchsorted(-n[order], -k, side="left")]   # rows of more than k entries
        q = ptr[r] + k
        with np.errstate(all="ignore"):
            s[r] = s[r] + val[q] * x[idx[q]]
    return s


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", [1, 2, 33, 1183, 1184, 1185, 40000, "full-1", "full", "full+1"])
def test_sums_in_storage_order(cuda, kind, dtype):
    import torch
    n, rng = lengths(kind), np.random.default_rng(11)
    ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    cols = 5003
    idx = rng.integers(0, cols, ptr[-1]).astype(np.int32)
    val = rng.standard_normal(ptr[-1]).astype(dtype)
    x = rng.standard_normal(cols).astype(dtype)
    x[5], x[6], x[7] = np.inf, np.nan, -0.0
    val[:3] = [0.0, -0.0, np.inf][: min(3, val.size)]
    t = [torch.from_numpy(a).cuda() for a in (ptr, idx, val, x)]
    out = torch.full((n.size,), 7.0, dtype=t[2].dtype, device="cuda")
    name = "f64" if dtype == np.float64 else "f32"
    for call in ("vajra_csr_spmv_", "vajra_csc_spmv_transpose_"):
        out.fill_(7.0)
        torch.cuda.synchronize()
        p = [C.c_void_p(a.data_ptr()) for a in (*t, out)]
        assert getattr(_capi.lib(), call + name)(n.size, *p, None) == 0
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), in_order(ptr, idx, val, x), err_msg=call)


def test_reference_algorithm_with_full_ctas_equals_the_oracle(cuda):
    """Columns enough for CTAs of 256, one to six entries each; x_bar entries of at most 1e-11 left out."""
    from oracle import bindings as B
    lp = W.random_planted(2000, FULL + 99, (1, 6), seed=8)
    kw = dict(iteration_limit=12, check_frequency=5, tolerance=1e-9, gap_tolerance=1e-9)
    g, o = V.solve(lp, algorithm=V.ALGO_REFERENCE, **kw), B.port_solve(lp, **kw)
    for k in ("x", "y", "d", "row_value"):
        np.testing.assert_array_equal(g[k], o[k], err_msg=k)
    assert g["iterations"] == o["iterations"] and g["objective_value"] == o["objective_value"]
