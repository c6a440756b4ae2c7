"""Performance cases of the LP framework: what its users have it do, over the sizes they do it at.

Every case goes through the public Python entry points (``solve``, ``Solver.run``, ``solve_batch``,
``autograd.unrolled``) or the device-pointer C entry points, on LPs of ``vajra_pdhg.workloads``.
``exact`` restates each path in 64 bits with plain torch.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vajra-opt_b200"))
import vajra_pdhg as V  # noqa: E402
from vajra_pdhg import _capi, autograd, workloads as W  # noqa: E402

# The autotuner runs on matrices of this many entries and more.  It picks launch shapes by
# timing, and FP32 row sums round by shape: where a case iterates in FP32 on such a matrix it
# fixes the shapes (-3, sliced ELL), as a program does that wants repeatable results.
TUNED_NNZ = 1 << 20


def listed():
    return [
        # One call on a textbook-size LP (a Netlib-size model inside an application): everything
        # is latency -- upload, set-up launches, a few hundred iterations, download.
        {"name": "call_tiny", "kind": "call", "lp": "planted", "m": 60, "n": 150, "klo": 4, "khi": 4,
         "precision": "mixed", "tol": 1e-6, "limit": 20000},
        # One call on a small LP to 1e-6, default options (the 2,000 x 5,000 workload).
        {"name": "call_small", "kind": "call", "lp": "planted", "m": 2000, "n": 5000, "klo": 8, "khi": 8,
         "precision": "mixed", "tol": 1e-6, "limit": 20000},
        # A resident model with ==, <=, >= and ranged rows solved again in plain FP64.
        {"name": "resident_senses", "kind": "resident", "lp": "senses", "m": 301, "n": 807, "klo": 3, "khi": 3,
         "precision": "fp64", "tol": 1e-6, "limit": 4000},
        # A mid-size LP, ragged column lengths, plain FP64, to 1e-4 (a warm start for a crossover).
        {"name": "resident_mid", "kind": "resident", "lp": "planted", "m": 20011, "n": 50021, "klo": 4, "khi": 12,
         "precision": "fp64", "tol": 1e-4, "limit": 4096},
        # Min-cost flow, 200k nodes x 1.5M arcs: two entries a column, plain FP64.
        {"name": "flow", "kind": "resident", "lp": "flow", "m": 200_000, "n": 1_500_000, "klo": 2, "khi": 2,
         "precision": "fp64", "tol": 1e-9, "limit": 1024},
        # The 1M x 2M heavy-tailed LP in mixed precision: a fixed budget of iterations.
        {"name": "large_mixed", "kind": "resident", "lp": "large", "m": 1_000_000, "n": 2_000_000, "klo": 2,
         "khi": 2000, "precision": "mixed", "tol": 1e-9, "limit": 1024},
        # Half that size in plain FP64 as one cold call: upload, ordering, iterations, download.
        {"name": "call_large_fp64", "kind": "call", "lp": "large", "m": 500_000, "n": 1_000_000, "klo": 2,
         "khi": 2000, "precision": "fp64", "tol": 1e-9, "limit": 512},
        # Many small LPs in one batched call to 1e-4, mixed precision, shapes by the heuristic.
        {"name": "batch_small", "kind": "batch", "lp": "planted", "count": 96, "m": 100, "n": 2000, "klo": 4,
         "khi": 12, "precision": "mixed", "tol": 1e-4, "limit": 6000},
        # The uneven batch (m log-uniform on [100, 20,000]) in plain FP64, a budget of iterations.
        {"name": "batch_uneven", "kind": "batch", "lp": "planted", "count": 256, "m": 100, "n": 20_000, "klo": 4,
         "khi": 12, "precision": "fp64", "tol": 1e-9, "limit": 1000},
        # Forward and backward of the unrolled map over a batch (learning c and b), mixed precision.
        {"name": "unrolled", "kind": "unrolled", "lp": "planted", "count": 32, "m": 1000, "n": 3000, "klo": 8,
         "khi": 8, "precision": "mixed", "limit": 1000},
        # The reference algorithm, bit for bit, as the drop-in runs it by default.
        {"name": "reference", "kind": "reference", "lp": "planted", "m": 2000, "n": 5000, "klo": 8, "khi": 8,
         "precision": "fp64", "tol": 1e-6, "limit": 2000},
        # A caller's own PDHG loop on device arrays: four fused steps, the relative KKT, the
        # residual diagnostics.
        {"name": "device_steps", "kind": "steps", "lp": "planted", "m": 100_003, "n": 250_007, "klo": 4, "khi": 12,
         "precision": "fp64", "limit": 4},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "call", "resident", "resident", "batch", "unrolled", "reference", "steps"])
    precision = rng.choice(["mixed", "fp64"])
    klo = rng.randint(2, 6)
    case = {"kind": kind, "lp": "planted", "klo": klo, "khi": klo + rng.randint(0, 8), "precision": precision}
    if kind in ("call", "resident"):
        m = log_int(40, 300_000)
        lp = rng.choice(["planted", "planted", "senses", "flow", "large"])
        if lp in ("flow", "large"):
            m = log_int(1000, 150_000)
        n = round(rng.uniform(5.0, 8.0) * m) if lp == "flow" else round(rng.uniform(2.0, 3.0) * m)
        case.update(lp=lp, m=m, n=n, tol=1e-6 if m < 10_000 else 1e-9, limit=4000 if m < 10_000 else 500)
    elif kind == "batch":
        m = log_int(30, 1000)
        case.update(count=log_int(4, 128), m=m, n=round(m * rng.uniform(1.5, 8.0)), tol=1e-9, limit=rng.randint(500, 2000))
    elif kind == "unrolled":
        case.update(count=log_int(1, 48), m=log_int(40, 2000), limit=rng.randint(100, 700))
        case["n"] = round(rng.uniform(2.0, 3.0) * case["m"])
    elif kind == "reference":
        m = log_int(40, 6000)
        case.update(m=m, n=round(rng.uniform(2.0, 3.0) * m), precision="fp64", tol=1e-6, limit=rng.randint(300, 1500))
    else:
        m = log_int(100, 200_000)
        case.update(m=m, n=round(rng.uniform(2.0, 3.0) * m), precision="fp64", limit=rng.randint(1, 8))
    return case


# ----- inputs -------------------------------------------------------------------------------
def _one_lp(case, m, n, seed):
    k = (case["klo"], min(case["khi"], m))
    if case["lp"] == "flow":
        return W.min_cost_flow(m, n, seed=seed)
    if case["lp"] == "large":
        return W.random_large(m, n, seed=seed, kmin=2, kmax=min(2000, m // 2))
    if case["lp"] == "senses":
        return W.small_random(m, n, seed=seed, density_per_col=case["klo"])
    return W.random_planted(m, n, k, seed=seed)


def _lps(case, seed):
    """The LPs of a case.  The sizes belong to the case; the entries and vectors to the seed."""
    if case["kind"] == "batch":   # m log-uniform on [case m, case n]
        sizes = W.batch_sizes(case["count"], seed=case["count"], m_lo=case["m"], m_hi=case["n"])
        return [_one_lp(case, m, n, seed * 100_003 + i) for i, (m, n, _) in enumerate(sizes)]
    return [_one_lp(case, case["m"], case["n"], seed * 1009 + i) for i in range(case.get("count", 1))]


def _precision(case):
    return V.PREC_FP64 if case["precision"] == "fp64" else V.PREC_MIXED


def _options(case, lps):
    if case["kind"] == "unrolled":
        return {"iterations": case["limit"], "checkpoint_every": 100, "precision": _precision(case)}
    o = {"tolerance": case["tol"], "iteration_limit": case["limit"]}
    if case["kind"] == "reference":
        return {**o, "algorithm": V.ALGO_REFERENCE, "check_frequency": 100}
    o["precision"] = _precision(case)
    if case["precision"] == "mixed":
        if case["kind"] == "batch":
            o["autotune"] = 0
        elif lps[0].nnz >= TUNED_NNZ:
            o.update(autotune=0, spmv_shape_a=-3, spmv_shape_at=-3)
    return o


def _device_lp(lp, seed):
    """A caller's own device copy of an LP: CSR and CSC, vectors, a point, step sizes."""
    rows = lp.row_idx.astype(np.int64)
    cols = np.repeat(np.arange(lp.num_cols, dtype=np.int64), np.diff(lp.col_ptr))
    order = torch.argsort(torch.from_numpy(rows * lp.num_cols + cols).cuda())
    g = {"row_ptr": np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=lp.num_rows))]).astype(np.int64),
         "col_ptr": lp.col_ptr, "row_idx": lp.row_idx, "csc": lp.values, "c": lp.c, "cl": lp.col_lower,
         "cu": lp.col_upper, "rl": lp.row_lower, "ru": lp.row_upper}
    d = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in g.items()}
    d["col_idx"] = torch.from_numpy(cols.astype(np.int32)).cuda()[order].contiguous()
    d["csr"] = d["csc"][order].contiguous()
    rng = np.random.default_rng(seed + 77)
    x = rng.uniform(0.0, 10.0, lp.num_cols)
    for k, v in (("x", x), ("xb", x), ("y", rng.standard_normal(lp.num_rows)), ("w", np.zeros(lp.num_rows)),
                 ("v", np.zeros(lp.num_cols)), ("kkt", np.zeros(6)), ("diag", np.zeros(6))):
        d[k] = torch.from_numpy(v.copy()).cuda()
    d["step"] = 0.5 / math.sqrt(float(np.abs(lp.values).max()) ** 2 * np.diff(g["row_ptr"]).max())
    return d


def prepare(case, seed):
    lps = _lps(case, seed)
    state = {"case": case, "lps": lps, "opts": _options(case, lps) if case["kind"] != "steps" else None}
    if case["kind"] == "resident":
        state["solver"] = V.Solver(lps[0], **state["opts"])
    elif case["kind"] == "unrolled":
        rng = np.random.default_rng(seed + 5)
        state["weights"] = rng.standard_normal(sum(lp.num_cols for lp in lps))
    elif case["kind"] == "steps":
        state["dev"] = _device_lp(lps[0], seed)
    return state


# ----- one pass -----------------------------------------------------------------------------
KEYS = ("x", "y", "row_value", "d")


def _solution(r):
    return {**{k: r[k] for k in KEYS}, "objective": float(r["objective_value"]), "iterations": int(r["iterations"]),
            "status": int(r["status"])}


def run(state):
    kind = state["case"]["kind"]
    if kind in ("call", "reference"):
        return _solution(V.solve(state["lps"][0], **state["opts"]))
    if kind == "resident":
        return _solution(state["solver"].run())
    if kind == "batch":
        rs = V.solve_batch(state["lps"], **state["opts"])
        out = {k: np.concatenate([r[k] for r in rs]) for k in KEYS}
        out["objective"] = np.array([r["objective_value"] for r in rs])
        out["iterations"] = np.array([r["iterations"] for r in rs])
        out["status"] = np.array([r["status"] for r in rs])
        return out
    if kind == "unrolled":
        return autograd.unrolled(state["lps"], state["weights"], **state["opts"])
    d, lp, lib = state["dev"], state["lps"][0], _capi.lib()
    p = {k: C.c_void_p(t.data_ptr()) for k, t in d.items() if k != "step"}
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    m, n = lp.num_rows, lp.num_cols
    ok = 0
    for _ in range(state["case"]["limit"]):
        ok |= lib.vajra_pdhg_step_f64(m, n, p["row_ptr"], p["col_idx"], p["csr"], p["col_ptr"], p["row_idx"],
                                      p["csc"], p["rl"], p["ru"], p["c"], p["cl"], p["cu"], d["step"], d["step"],
                                      p["x"], p["xb"], p["y"], p["w"], p["v"], st)
    ok |= lib.vajra_relative_kkt_noalloc_f64(m, n, p["row_ptr"], p["col_idx"], p["csr"], p["col_ptr"], p["row_idx"],
                                             p["csc"], p["c"], p["cl"], p["cu"], p["rl"], p["ru"], p["x"], p["y"], 0,
                                             0.0, p["kkt"], st)
    ok |= lib.vajra_device_diagnostics_f64(m, n, p["w"], p["rl"], p["ru"], p["v"], p["c"], p["x"], p["y"], p["cl"],
                                           p["cu"], p["diag"], st)
    if ok:
        raise RuntimeError("a device entry point failed")
    return {"x": d["x"], "xb": d["xb"], "y": d["y"], "w": d["w"], "v": d["v"], "kkt": d["kkt"],
            "diag": d["diag"][:3]}


# ----- what a pass cannot do without ----------------------------------------------------------
def work(case):
    """Iterations times one reading of A, A^T and the vectors (a solve to tolerance: a quarter of
    its limit), and the LP read and the results written once."""
    if case["kind"] == "batch":
        sizes = W.batch_sizes(case["count"], seed=case["count"], m_lo=case["m"], m_hi=case["n"])
    else:
        sizes = [(case["m"], case["n"], None)] * case.get("count", 1)
    m, n = sum(s[0] for s in sizes), sum(s[1] for s in sizes)
    mean = {"flow": 2.0, "large": 10.0, "senses": case["klo"]}.get(case["lp"], 0.5 * (case["klo"] + case["khi"]))
    nnz = mean * n
    t = 4 if case["precision"] == "mixed" and case["kind"] != "unrolled" else 8
    its = case["limit"] if case.get("tol", 0.0) < 1e-8 else max(64, case["limit"] // 4)
    if case["kind"] == "reference":
        its = case["limit"]
    per_it = 2.0 * (4 + t) * nnz + 6.0 * t * n + 5.0 * t * m
    passes = 3.0 if case["kind"] == "unrolled" else 1.0   # forward, recomputed forward, reverse
    return {"bytes": passes * its * per_it + 12.0 * nnz + 40.0 * n + 32.0 * m, "flops": passes * its * 4.0 * nnz}


# ----- the same paths in 64 bits ---------------------------------------------------------------
INF = 1e20


class _Packed:
    """Instances side by side as one block-diagonal LP in float64 on the GPU."""

    def __init__(self, lps):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda v, dt=torch.float64: torch.from_numpy(np.ascontiguousarray(v)).to(dev, dt)  # noqa: E731
        roff = np.concatenate([[0], np.cumsum([lp.num_rows for lp in lps])])
        coff = np.concatenate([[0], np.cumsum([lp.num_cols for lp in lps])])
        self.count, self.m, self.n = len(lps), int(roff[-1]), int(coff[-1])
        cat = lambda f: np.concatenate([f(i, lp) for i, lp in enumerate(lps)])  # noqa: E731
        self.row = t(cat(lambda i, lp: lp.row_idx.astype(np.int64) + roff[i]), torch.int64)
        self.col = t(cat(lambda i, lp: np.repeat(np.arange(lp.num_cols), np.diff(lp.col_ptr)) + coff[i]), torch.int64)
        self.val0 = t(cat(lambda i, lp: lp.values))
        self.c0, self.cl0, self.cu0 = (t(cat(lambda i, lp: getattr(lp, k))) for k in ("c", "col_lower", "col_upper"))
        self.rl0, self.ru0 = (t(cat(lambda i, lp: getattr(lp, k))) for k in ("row_lower", "row_upper"))
        self.ri = torch.repeat_interleave(torch.arange(self.count, device=dev), t(np.diff(roff), torch.int64))
        self.ci = torch.repeat_interleave(torch.arange(self.count, device=dev), t(np.diff(coff), torch.int64))
        self.by_row = torch.argsort(self.row * self.n + self.col)
        self.ptr_r = self._ptr(self.row, self.m)
        self.ptr_c = self._ptr(self.col, self.n)

    @staticmethod
    def _ptr(key, size):
        return torch.cat([key.new_zeros(1), torch.cumsum(torch.bincount(key, minlength=size), 0)])

    def scale(self, pock_chambolle, per_instance):
        row, col = self.row, self.col
        val, rs, cs = self.val0.clone(), torch.ones_like(self.rl0), torch.ones_like(self.c0)
        gi = lambda i: i if per_instance else torch.zeros_like(i)  # noqa: E731
        done = torch.zeros(self.count, dtype=torch.bool, device=val.device)
        factor = lambda v: torch.where(v > 1e-11, 1.0 / torch.sqrt(v.clamp_min(1e-300)), torch.ones_like(v))  # noqa: E731
        for _ in range(10):
            rn = torch.zeros_like(rs).scatter_reduce_(0, row, val.abs(), "amax")
            cn = torch.zeros_like(cs).scatter_reduce_(0, col, val.abs(), "amax")
            off = lambda v, i: torch.zeros(self.count, dtype=v.dtype, device=v.device).scatter_reduce_(  # noqa: E731
                0, gi(i), torch.where(v > 1e-11, (1.0 - v).abs(), torch.zeros_like(v)), "amax")
            done = done | ((off(rn, self.ri) <= 0.05) & (off(cn, self.ci) <= 0.05))
            r = torch.where(done[gi(self.ri)], torch.ones_like(rn), factor(rn))
            c = torch.where(done[gi(self.ci)], torch.ones_like(cn), factor(cn))
            rs, cs, val = rs * r, cs * c, val * (r[row] * c[col])
        if pock_chambolle:
            r = factor(torch.zeros_like(rs).scatter_add_(0, row, val.abs()))
            c = factor(torch.zeros_like(cs).scatter_add_(0, col, val.abs()))
            rs, cs, val = rs * r, cs * c, val * (r[row] * c[col])
        self.rs, self.cs, self.val = rs, cs, val
        self.c = self.c0 * cs
        keep = lambda v, s: torch.where(v.abs() < INF, v * s, v)  # noqa: E731
        self.cl, self.cu = keep(self.cl0, 1.0 / cs), keep(self.cu0, 1.0 / cs)
        self.rl, self.ru = keep(self.rl0, rs), keep(self.ru0, rs)
        self.a = torch.sparse_csr_tensor(self.ptr_r, self.col[self.by_row], val[self.by_row], (self.m, self.n))
        self.at = torch.sparse_csr_tensor(self.ptr_c, self.row, val, (self.n, self.m))
        self.a0 = torch.sparse_csr_tensor(self.ptr_r, self.col[self.by_row], self.val0[self.by_row], (self.m, self.n))
        self.at0 = torch.sparse_csr_tensor(self.ptr_c, self.row, self.val0, (self.n, self.m))

    def sum_c(self, v):
        return torch.zeros(self.count, dtype=v.dtype, device=v.device).index_add_(0, self.ci, v)

    def sum_r(self, v):
        return torch.zeros(self.count, dtype=v.dtype, device=v.device).index_add_(0, self.ri, v)

    def norm_rounds(self, rounds):
        v = 1.0 / torch.sqrt(self.sum_c(torch.ones_like(self.c)))[self.ci]
        for _ in range(rounds):
            u = self.at @ (self.a @ v)
            nrm = torch.sqrt(self.sum_c(u * u))
            v = u / nrm[self.ci]
        return torch.sqrt(nrm)

    def norm_to(self, rounds, tol):
        v = torch.full_like(self.c, 1.0 / math.sqrt(self.n))
        prev = 0.0
        for it in range(rounds):
            u = self.at @ (self.a @ v)
            nrm = float(torch.linalg.norm(u))
            if it > 0 and abs(nrm - prev) <= tol * nrm:
                break
            prev = nrm
            v = u / nrm
        return torch.full((self.count,), math.sqrt(nrm), dtype=v.dtype, device=v.device)

    def b_norm(self, lo, up):
        lf, uf = lo > -INF, up < INF
        z = torch.zeros_like(lo)
        both = torch.where(lf, lo * lo, z) + torch.where(uf, up * up, z)
        return torch.sqrt(self.sum_r(torch.where(lf & uf & (lo == up), lo * lo, both)))

    def solution(self, x, y, per_instance):
        out = {"x": x, "y": y, "row_value": self.a0 @ x, "d": self.c0 - self.at0 @ y}
        obj = self.sum_c(self.c0 * x)
        out["objective"] = obj.cpu() if per_instance else float(obj[0])
        out["iterations"] = out["status"] = None
        return {k: v.cpu() if isinstance(v, torch.Tensor) else v for k, v in out.items()}


def _halpern(lps, case):
    """The restarted reflected Halpern iteration, every instance with its own steps and restarts."""
    batch = case["kind"] == "batch"
    P = _Packed(lps)
    P.scale(True, True)
    eta = 0.99 / (P.norm_rounds(60) if batch else P.norm_to(100, 1e-5))
    csn, bsn = torch.sqrt(P.sum_c(P.c * P.c)), P.b_norm(P.rl, P.ru)
    omega = torch.where((csn > 1e-10) & (bsn > 1e-10), csn / bsn, torch.ones_like(csn))
    cn, bn = torch.sqrt(P.sum_c(P.c0 * P.c0)), P.b_norm(P.rl0, P.ru0)
    tau, sigma = eta / omega, eta * omega
    x = torch.zeros_like(P.c).clamp(P.cl, P.cu)
    y = torch.zeros_like(P.rl)
    x0, y0, xl, yl, xc, yc = x, y, x, y, x, y
    k, total = torch.zeros_like(eta), torch.zeros_like(eta)
    start, prev = torch.full_like(eta, -1.0), torch.full_like(eta, -1.0)
    done = torch.zeros(P.count, dtype=torch.bool, device=x.device)
    lf, uf, rlf, ruf = P.cl0 > -INF, P.cu0 < INF, P.rl0 > -INF, P.ru0 < INF
    zr, zc = torch.zeros_like(y), torch.zeros_like(x)
    lam_of = lambda r: torch.where(lf & uf, r, torch.where(lf, r.clamp_min(0), torch.where(uf, r.clamp_max(0), zc)))  # noqa: E731
    left = case["limit"]
    while left > 0 and not bool(done.all()):
        ln = min(64, left)
        left -= ln
        on_c, on_r = ~done[P.ci], ~done[P.ri]
        tc, sr = tau[P.ci], sigma[P.ri]
        for kk in range(ln):
            w1, w0 = (k + kk + 1) / (k + kk + 2), 1.0 / (k + kk + 2)
            xp = torch.minimum(torch.maximum(x - tc * (P.c + P.at @ y), P.cl), P.cu)
            yh = y + sr * (P.a @ (2 * xp - x))
            yp = yh - sr * torch.minimum(torch.maximum(yh / sr, P.rl), P.ru)
            x = torch.where(on_c, w1[P.ci] * (2 * xp - x) + w0[P.ci] * x0, x)
            y = torch.where(on_r, w1[P.ri] * (2 * yp - y) + w0[P.ri] * y0, y)
        xc, yc = torch.where(on_c, xp, xc), torch.where(on_r, yp, yc)
        ax, aty = P.a @ xc, P.at @ yc
        total = total + torch.where(done, 0.0, float(ln))
        ao, yo = ax / P.rs, -yc * P.rs
        rp = torch.sqrt(P.sum_r((ao - torch.minimum(torch.maximum(ao, P.rl0), P.ru0)) ** 2))
        rps2 = P.sum_r((ax - torch.minimum(torch.maximum(ax, P.rl), P.ru)) ** 2)
        dr = P.sum_r(torch.where((yo > 0) & rlf, yo * P.rl0, torch.where((yo < 0) & ruf, yo * P.ru0, zr)))
        r_s = P.c + aty
        r_o = r_s / P.cs
        lo, ls = lam_of(r_o), lam_of(r_s)
        rd, rds2 = torch.sqrt(P.sum_c((r_o - lo) ** 2)), P.sum_c((r_s - ls) ** 2)
        dobj = dr + P.sum_c(torch.where(lo > 0, lo * P.cl0, torch.where(lo < 0, lo * P.cu0, zc)))
        pobj = P.sum_c(P.c * xc)
        gap = (pobj - dobj).abs() / (1 + pobj.abs() + dobj.abs())
        rel = torch.maximum(rp / (1 + bn), torch.maximum(rd / (1 + cn), gap))
        done = done | (rel <= case["tol"])
        wk = torch.sqrt(omega * rps2 + rds2 / omega + gap * gap)
        first = start < 0
        start, prev = torch.where(first, wk, start), torch.where(first, wk, prev)
        again = ~done & ((wk <= 0.2 * start) | ((wk <= 0.8 * start) & (wk > prev)) | (k + ln >= 0.36 * total))
        prev = wk
        dx, dy = torch.sqrt(P.sum_c((xc - xl) ** 2)), torch.sqrt(P.sum_r((yc - yl) ** 2))
        move = again & (dx > 1e-10) & (dy > 1e-10)
        omega = torch.where(move, torch.exp(0.5 * torch.log(dy.clamp_min(1e-300) / dx.clamp_min(1e-300)) + 0.5 * torch.log(omega)), omega)
        tau, sigma = eta / omega, eta * omega
        k = torch.where(again, torch.zeros_like(k), k + ln)
        start = torch.where(again, wk, start)
        ac, ar = again[P.ci], again[P.ri]
        x, x0, xl = torch.where(ac, xc, x), torch.where(ac, xc, x0), torch.where(ac, xc, xl)
        y, y0, yl = torch.where(ar, yc, y), torch.where(ar, yc, y0), torch.where(ar, yc, yl)
    return P.solution(xc * P.cs, -yc * P.rs, batch)


def _reference(lps, case):
    """The reference algorithm: dual first, residual checks, step rebalancing, best iterate."""
    P = _Packed(lps)
    P.scale(False, False)
    norm = float(P.norm_to(25, 1e-4)[0])
    tau = sigma = 0.95 / norm
    drop = lambda v: torch.where(v.abs() <= 1e-11, torch.zeros_like(v), v)  # noqa: E731
    x = torch.zeros_like(P.c).clamp(P.cl, P.cu)
    y = torch.zeros_like(P.rl)
    xb, bx, by, best, idle = x, x, y, 1e20, 0
    for it in range(1, case["limit"] + 1):
        yh = y + sigma * (P.a @ drop(xb))
        y = yh - sigma * torch.minimum(torch.maximum(yh / sigma, P.rl), P.ru)
        v = P.at @ y
        xn = torch.minimum(torch.maximum(x - tau * (v + P.c), P.cl), P.cu)
        xb, x = 2 * xn - x, xn
        if it % 100 and it != case["limit"]:
            continue
        ax, d = P.a @ drop(x), P.c + v
        prim = float(torch.maximum(P.rl - ax, ax - P.ru).clamp_min(0).max())
        up, dn = d[(x > P.cl + 1e-5) & (d > 1e-6)], -d[(x < P.cu - 1e-5) & (d < -1e-6)]
        free = d[(P.cl <= -INF) & (P.cu >= INF)].abs()
        dual = max([0.0] + [float(q.max()) for q in (up, dn, free) if q.numel()])
        z, zc = torch.zeros_like(y), torch.zeros_like(x)
        dob = float((torch.where((y > 1e-12) & (P.ru < INF), -y * P.ru, torch.where((y < -1e-12) & (P.rl > -INF), -y * P.rl, z))).sum()
                    + (torch.where((d > 1e-12) & (P.cl > -INF), d * P.cl, torch.where((d < -1e-12) & (P.cu < INF), d * P.cu, zc))).sum())
        pob = float((P.c * x).sum())
        if prim + dual < best:
            best, idle, bx, by = prim + dual, 0, x, y
        else:
            idle += 100
        if prim <= case["tol"] and dual <= case["tol"] and abs(pob - dob) / (1 + abs(pob) + abs(dob)) <= 1e-6:
            bx, by = x, y
            break
        if prim > 10 * dual and dual > 0:
            sigma = min(sigma * 1.3, 1e6)
            tau = 0.95 ** 2 / (norm * norm * sigma)
        elif dual > 10 * prim and prim > 0:
            tau = min(tau * 1.3, 1e6)
            sigma = 0.95 ** 2 / (norm * norm * tau)
        if idle >= 200:
            xb, idle = x, 0
    return P.solution(bx * P.cs, -by * P.rs, False)


def _unrolled(lps, case, weights):
    P = _Packed(lps)
    P.scale(True, False)
    step = 0.95 / P.norm_rounds(60)
    tc, sr = step[P.ci], step[P.ri]
    x = torch.zeros_like(P.c).clamp(P.cl, P.cu)
    y = torch.zeros_like(P.rl)
    inside, code = [], []
    for _ in range(case["limit"]):
        pre = x - tc * (P.c + P.at @ y)
        xn = torch.minimum(torch.maximum(pre, P.cl), P.cu)
        inside.append((pre > P.cl) & (pre < P.cu))
        q = y + sr * (P.a @ (2 * xn - x))
        t = q / sr
        code.append((t < P.rl).to(torch.int8) + 2 * (t > P.ru).to(torch.int8))
        y = q - sr * torch.minimum(torch.maximum(t, P.rl), P.ru)
        x = xn
    w = torch.from_numpy(weights).to(x) + P.c0
    xh, yh = P.cs * w, torch.zeros_like(y)
    gc, gl, gu = torch.zeros_like(x), torch.zeros_like(y), torch.zeros_like(y)
    for p, cd in zip(reversed(inside), reversed(code)):
        gl, gu = gl - sr * yh * (cd == 1), gu - sr * yh * (cd == 2)
        q = yh * (cd != 0)
        xbh = P.at @ (sr * q)
        pre = (xh + 2 * xbh) * p
        gc = gc - tc * pre
        xh, yh = pre - xbh, q - sr * (P.a @ pre)
    xo = P.cs * x
    return {"loss": P.sum_c(w * xo).cpu(), "x": xo.cpu(), "grad_c": (P.cs * gc + xo).cpu(),
            "grad_row_lower": torch.where(P.rl0 > -INF, P.rs * gl, 0 * gl).cpu(),
            "grad_row_upper": torch.where(P.ru0 < INF, P.rs * gu, 0 * gu).cpu()}


def _steps(lp, seed, case):
    d = _device_lp(lp, seed)
    P = _Packed([lp])
    P.scale(False, False)
    A, At, s = P.a0, P.at0, d["step"]
    x, xb, y = d["x"], d["xb"], d["y"]
    for _ in range(case["limit"]):
        w = A @ xb
        yh = y + s * w
        y = yh - s * torch.minimum(torch.maximum(yh / s, P.rl0), P.ru0)
        v = At @ y
        xn = torch.minimum(torch.maximum(x - s * (v + P.c0), P.cl0), P.cu0)
        xb, x = 2 * xn - x, xn
    # every row an equality, every column boxed
    ax, r = A @ x, P.c0 - At @ y
    lam = r
    rp = float(torch.linalg.norm(ax - P.rl0) / (1 + torch.linalg.norm(P.rl0)))
    pobj = float((P.c0 * x).sum())
    dobj = float((y * P.rl0).sum() + torch.where(lam > 0, lam * P.cl0, lam * P.cu0).sum())
    gap = abs(pobj - dobj) / (1 + abs(pobj) + abs(dobj))
    rc = P.c0 + v
    prim = max(float((w - P.rl0).abs().max()), float(torch.maximum(P.cl0 - x, x - P.cu0).max()), 0.0)
    bad = torch.where((x < P.cu0 - 1e-5) & (rc < -1e-6), -rc, torch.where((x > P.cl0 + 1e-5) & (rc > 1e-6), rc, 0 * rc))
    out = {"x": x, "xb": xb, "y": y, "w": w, "v": v,
           "kkt": torch.tensor([rp, 0.0, gap, max(rp, gap), pobj, dobj], dtype=torch.float64),
           "diag": torch.tensor([prim, float(bad.max()), pobj], dtype=torch.float64)}
    return {k: t.cpu() for k, t in out.items()}


def exact(case, seed):
    lps = _lps(case, seed)
    kind = case["kind"]
    if kind == "unrolled":
        w = np.random.default_rng(seed + 5).standard_normal(sum(lp.num_cols for lp in lps))
        return _unrolled(lps, case, w)
    if kind == "reference":
        return _reference(lps, case)
    if kind == "steps":
        return _steps(lps[0], seed, case)
    if case["precision"] == "mixed" and case["tol"] > 1e-8:
        # solved to tolerance from FP32 iterates: the optimal objective is the one exact value
        known = [lp.planted_objective for lp in lps]
        if any(v is None for v in known):
            return None
        out = dict.fromkeys(KEYS + ("iterations", "status"))
        out["objective"] = np.array(known) if kind == "batch" else float(known[0])
        return out
    return _halpern(lps, case)
