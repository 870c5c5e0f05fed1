"""The work this engine is timed on, through its public entry points.

Every case is one of eight kinds of call that a user's program makes:

  call     solve_pdhg_gpu(lp, options, engine=engine): the whole seam call of one LP (load,
           preconditioning, iterations, read-back) on an engine that the program keeps, as
           SANKHYA's solve() makes it
  solve    PdhgEngine.solve + solution on an LP loaded before: re-solves of a large LP
  product  PdhgEngine.spmv_device: A x and A'y on the caller's device buffers
  scaling  PdhgEngine.scaling: the preconditioner and the spectral norm, the setup of every solve
  qp       QpEngine.solve + solution on a QP loaded before
  qpcall   solve_convex_qp_gpu(qp, options, engine=engine): the whole QP call
  nodes    BatchEngine.load + solve + solution: branch-and-bound node relaxations that share
           one matrix
  backward BatchEngine.polish + adjoint + solution: the vertices and the gradients of a batch
           of LPs from the points that a forward pass left

LPs and QPs come from the repository's own seeded generators, at the shapes of its tests and
its benchmark (planted uniform, block-angular, Zipf-row, general and nondegenerate LPs; banded
Hessians).

FP64 solves stop at an iteration limit (branch-and-bound probes and time-sliced solves run this
way). PDHG's adaptive step size feeds every rounding error back into the trajectory: on these
LPs a last-bit change of the data moves the point by 1e-12 after two evaluation periods (80
iterations) and by 1e-6 to 1e-3 after twenty, so the limits are a few evaluation periods, each
with its restart tests, evaluations and candidate selection. The convex-QP iteration has a fixed
step and no such feedback, so QPs run for hundreds or thousands.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "sih-26_gb300"))
from sankhya_gb300 import capi, lpgen  # noqa: E402
from sankhya_gb300.model import LP, QP, banded_hessian  # noqa: E402

PERIOD_ROWS, PERIOD_COLS = 15625, 31250  # one period of the block-angular LP


def listed():
    return [
        # The smallest seam call: a few launches' worth of arithmetic, all latency.
        {"name": "call fp64 50x100", "kind": "call", "family": "uniform", "rows": 50,
         "cols": 100, "per_col": 5, "precision": "fp64", "iterations": 80},
        # The parity-sized seam call, every row and column kind, odd sizes, maximisation.
        {"name": "call fp64 general 1999x4001", "kind": "call", "family": "general",
         "rows": 1999, "cols": 4001, "per_col": 4, "precision": "fp64", "iterations": 80},
        # The block-angular multi-period LP in FP64, resident in HBM.
        {"name": "solve fp64 blocks 500k x 1M", "kind": "solve", "family": "blocks",
         "rows": 32 * PERIOD_ROWS, "cols": 32 * PERIOD_COLS, "per_col": 9, "periods": 32,
         "precision": "fp64", "iterations": 120},
        # The headline solve: 64 periods in the mixed method.
        {"name": "solve mixed blocks 1M x 2M", "kind": "solve", "family": "blocks",
         "rows": 64 * PERIOD_ROWS, "cols": 64 * PERIOD_COLS, "per_col": 9, "periods": 64,
         "precision": "mixed", "iterations": 800},
        # Load-balance stress: Zipf row lengths up to thousands of entries, scattered columns.
        {"name": "solve fp64 zipf 50k x 100k", "kind": "solve", "family": "zipf",
         "rows": 50000, "cols": 100000, "per_col": 30, "precision": "fp64", "iterations": 80},
        # One product pair (A x and A'y) with a large scattered matrix.
        {"name": "product 300k x 600k", "kind": "product", "family": "uniform",
         "rows": 300001, "cols": 600007, "per_col": 5},
        # The setup of every solve: ten Ruiz rounds, Pock-Chambolle, thirty power steps.
        {"name": "scaling blocks 250k x 500k", "kind": "scaling", "family": "blocks",
         "rows": 16 * PERIOD_ROWS, "cols": 16 * PERIOD_COLS, "per_col": 9, "periods": 16},
        # The smallest QP call: the default tolerance, with the iteration limit that a program
        # sets so that a slow instance does not hold it up.
        {"name": "qpcall 60x120", "kind": "qpcall", "family": "general", "rows": 60,
         "cols": 120, "per_col": 4, "band": 2, "iterations": 2000},
        # A middling QP with scattered rows.
        {"name": "qp uniform 20k x 40k", "kind": "qp", "family": "uniform", "rows": 20000,
         "cols": 40000, "per_col": 5, "band": 2, "iterations": 1000},
        # The large QP: the block-angular LP's rows with a banded Hessian.
        {"name": "qp blocks 500k x 1M", "kind": "qp", "family": "blocks",
         "rows": 32 * PERIOD_ROWS, "cols": 32 * PERIOD_COLS, "per_col": 9, "periods": 32,
         "band": 2, "iterations": 500},
        # Node relaxations that share one matrix, one batched launch.
        {"name": "nodes 304 of 1000x2000", "kind": "nodes", "family": "uniform", "rows": 1000,
         "cols": 2000, "per_col": 5, "count": 304, "iterations": 80},
        # The backward direction: polish and implicit gradients of a differentiable LP layer.
        {"name": "backward 128 of 1000x2000", "kind": "backward", "family": "nondegenerate",
         "rows": 1000, "cols": 2000, "per_col": 5, "count": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "solve", "solve", "product", "scaling", "qpcall", "qp",
                       "qp", "nodes", "backward"])
    if kind in ("call", "solve"):
        precision = rng.choice(["fp64", "fp64", "mixed"])
        if kind == "call":
            family = rng.choice(["uniform", "general"])
            rows = _log_int(rng, 50, 20000)
            return {"kind": kind, "family": family, "rows": rows,
                    "cols": 2 * rows + rng.randrange(-rows // 4, rows),
                    "per_col": rng.randrange(3, 7), "precision": precision, "iterations": 80}
        family = rng.choice(["blocks", "blocks", "zipf", "uniform"])
        if family == "blocks":
            periods = _log_int(rng, 2, 24)
            r = _log_int(rng, 2000, PERIOD_ROWS)
            c = 2 * r + rng.randrange(0, 99)
            return {"kind": kind, "family": family, "rows": periods * r, "cols": periods * c,
                    "per_col": rng.randrange(6, 11), "periods": periods,
                    "precision": precision, "iterations": 80 if precision == "fp64" else 400}
        rows = _log_int(rng, 5000, 60000)
        return {"kind": kind, "family": family, "rows": rows, "cols": 2 * rows + 1,
                "per_col": rng.randrange(15, 31) if family == "zipf" else rng.randrange(4, 9),
                "precision": precision, "iterations": 80}
    if kind == "product":
        family = rng.choice(["uniform", "zipf", "general"])
        rows = _log_int(rng, 500, 200000 if family == "uniform" else 50000)
        return {"kind": kind, "family": family, "rows": rows,
                "cols": 2 * rows + rng.randrange(1, 100), "per_col": rng.randrange(4, 12)}
    if kind == "scaling":
        periods = _log_int(rng, 2, 16)
        r = _log_int(rng, 1000, PERIOD_ROWS)
        return {"kind": kind, "family": "blocks", "rows": periods * r,
                "cols": periods * (2 * r + 1), "per_col": rng.randrange(6, 11),
                "periods": periods}
    if kind == "qpcall":
        rows = _log_int(rng, 30, 500)
        return {"kind": kind, "family": rng.choice(["uniform", "general"]), "rows": rows,
                "cols": 2 * rows + rng.randrange(0, rows), "per_col": rng.randrange(3, 6),
                "band": rng.randrange(1, 4), "iterations": 2000}
    if kind == "qp":
        family = rng.choice(["blocks", "uniform", "zipf"])
        if family == "blocks":
            periods = _log_int(rng, 2, 24)
            r = _log_int(rng, 2000, PERIOD_ROWS)
            return {"kind": kind, "family": family, "rows": periods * r,
                    "cols": periods * (2 * r + rng.randrange(0, 99)),
                    "per_col": rng.randrange(6, 11), "periods": periods,
                    "band": rng.randrange(0, 4), "iterations": 250}
        rows = _log_int(rng, 1000, 60000)
        return {"kind": kind, "family": family, "rows": rows, "cols": 2 * rows + 3,
                "per_col": rng.randrange(15, 25) if family == "zipf" else rng.randrange(3, 9),
                "band": rng.randrange(0, 4), "iterations": 500}
    if kind == "nodes":
        rows = _log_int(rng, 100, 2500)
        return {"kind": kind, "family": "uniform", "rows": rows, "cols": 2 * rows + 1,
                "per_col": rng.randrange(4, 7), "count": rng.randrange(40, 400),
                "iterations": 80}
    rows = _log_int(rng, 50, 1000)
    return {"kind": kind, "family": "nondegenerate", "rows": rows,
            "cols": 2 * rows + rng.randrange(0, rows // 2), "per_col": rng.randrange(4, 7),
            "count": rng.randrange(8, 120)}


# ---- Inputs --------------------------------------------------------------------------------

def _lp(case, seed) -> LP:
    m, n, k = case["rows"], case["cols"], case["per_col"]
    family = case["family"]
    if family == "uniform":
        return lpgen.planted_uniform(m, n, k, seed=seed)
    if family == "general":
        return lpgen.planted_general(m, n, k, seed=seed, maximize=bool(seed & 1), free=False)
    if family == "blocks":
        p = case["periods"]
        return lpgen.planted_blocks(p, m // p, n // p, k, seed=seed)
    if family == "zipf":
        return lpgen.planted_zipf(m, n, k * n, seed=seed)
    if family == "nondegenerate":
        return lpgen.planted_nondegenerate(m, n, k, seed=seed)
    raise ValueError(family)


def _qp(case, seed) -> QP:
    lp = _lp(case, seed)
    starts, index, values = banded_hessian(lp.cols, case["band"], seed)
    return QP(lp, starts, index, lp.sense * values)


def _vectors(lp, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(lp.cols), rng.standard_normal(lp.rows)


def _node_bounds(lp, count, seed):
    """Branch-and-bound node bounds: 1 to 20 columns rounded down or up at the planted point."""
    rng = np.random.default_rng(seed)
    nodes = []
    for _ in range(count):
        lo, up = lp.col_lower.copy(), lp.col_upper.copy()
        for j in rng.choice(lp.cols, size=int(rng.integers(1, 21)), replace=False):
            if rng.random() < 0.5:
                up[j] = np.floor(lp.x0[j])
            else:
                lo[j] = np.ceil(lp.x0[j])
        nodes.append((lo, up))
    return nodes


def _backward_inputs(case, seed):
    lps = [lpgen.planted_nondegenerate(case["rows"], case["cols"], case["per_col"],
                                       seed=1000 * (seed % 100000) + k).contiguous()
           for k in range(case["count"])]
    rng = np.random.default_rng(seed)
    gx = rng.standard_normal((len(lps), case["cols"]))
    gy = rng.standard_normal((len(lps), case["rows"]))
    return lps, gx, gy


def _reduced(lp):
    """c - A'y at the planted multipliers."""
    cols = np.repeat(np.arange(lp.cols), np.diff(lp.col_starts))
    return lp.col_cost - np.bincount(cols, lp.values * lp.lam[lp.row_index], lp.cols)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("call", "solve", "product", "scaling"):
        s["lp"] = _lp(case, seed).contiguous()
        s["engine"] = capi.PdhgEngine(0)
        if kind != "call":
            s["engine"].load(s["lp"])
        if kind == "product":
            x, y = _vectors(s["lp"], seed)
            s["x"] = torch.as_tensor(x, device="cuda")
            s["y"] = torch.as_tensor(y, device="cuda")
            s["ax"] = torch.empty(s["lp"].rows, dtype=torch.float64, device="cuda")
            s["aty"] = torch.empty(s["lp"].cols, dtype=torch.float64, device="cuda")
    elif kind in ("qp", "qpcall"):
        s["qp"] = _qp(case, seed).contiguous()
        s["engine"] = capi.QpEngine(0)
        if kind == "qp":
            s["engine"].load(s["qp"])
    elif kind == "nodes":
        lp = _lp(case, seed).contiguous()
        s["lps"] = [LP(lp.rows, lp.cols, lp.col_starts, lp.row_index, lp.values, lp.col_cost,
                       lo, up, lp.row_lower, lp.row_upper)
                    for lo, up in _node_bounds(lp, case["count"], seed)]
        s["engine"] = capi.BatchEngine(0)
        # A program that wants the same bits on every run fixes the schedule.
        s["engine"].set_schedule(1, 512)
    else:
        # The forward pass leaves converged LPs; their points are then the known vertices, as a
        # program hands a parent's vertex to its children.
        lps, gx, gy = _backward_inputs(case, seed)
        s["lps"], s["gx"], s["gy"] = lps, list(gx), list(gy)
        s["engine"] = capi.BatchEngine(0)
        s["engine"].set_schedule(1, 256)
        s["engine"].load(lps)
        s["engine"].solve(tolerance=0.03, stop_rule="relative", iteration_limit=20000)
        for k, lp in enumerate(lps):
            s["engine"].set_point(k, lp.x0, _reduced(lp), lp.lam)
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "call":
        r = capi.solve_pdhg_gpu(s["lp"], {"pdhg_tolerance": 1e-9,
                                          "pdhg_precision": case["precision"],
                                          "iteration_limit": case["iterations"]},
                                engine=s["engine"])
        return {"x": r.col_value, "reduced": r.col_dual, "y": r.row_dual,
                "iterations": r.iterations, "objective": np.float64(r.objective)}
    if kind == "solve":
        r = s["engine"].solve(tolerance=1e-9, precision=case["precision"],
                              iteration_limit=case["iterations"])
        x, d, y = s["engine"].solution()
        return {"x": x, "reduced": d, "y": y, "iterations": r.iterations,
                "objective": np.float64(r.objective)}
    if kind == "product":
        stream = torch.cuda.current_stream().cuda_stream
        s["engine"].spmv_device(0, s["x"].data_ptr(), s["ax"].data_ptr(), stream=stream or None)
        s["engine"].spmv_device(1, s["y"].data_ptr(), s["aty"].data_ptr(), stream=stream or None)
        return {"ax": s["ax"], "aty": s["aty"]}
    if kind == "scaling":
        dr, dc, values, norm = s["engine"].scaling()
        return {"row_scale": dr, "col_scale": dc, "values": values, "norm": np.float64(norm)}
    if kind == "qp":
        r = s["engine"].solve(tolerance=1e-9, iteration_limit=case["iterations"])
        x, d, y = s["engine"].solution()
        return {"x": x, "reduced": d, "y": y, "iterations": r.iterations,
                "objective": np.float64(r.objective)}
    if kind == "qpcall":
        r = capi.solve_convex_qp_gpu(s["qp"], {"iteration_limit": case["iterations"]},
                                     engine=s["engine"])
        return {"x": r.col_value, "reduced": r.col_dual, "y": r.row_dual,
                "iterations": r.iterations, "objective": np.float64(r.objective)}
    if kind == "nodes":
        eng = s["engine"]
        eng.load(s["lps"])
        items, _ = eng.solve(tolerance=1e-9, iteration_limit=case["iterations"])
        points = [eng.solution(k) for k in range(len(items))]
        return {"x": np.stack([p[0] for p in points]), "reduced": np.stack([p[1] for p in points]),
                "y": np.stack([p[2] for p in points]),
                "iterations": np.array([it.iterations for it in items]),
                "objective": np.array([it.objective for it in items])}
    eng = s["engine"]
    items, _ = eng.polish()
    grads = eng.adjoint(s["gx"], s["gy"], np.ones(len(items)))
    points = [eng.solution(k) for k in range(len(items))]
    return {"x": np.stack([p[0] for p in points]), "y": np.stack([p[2] for p in points]),
            "f": np.array([it.objective for it in items]),
            "status": np.array([g["status"] for g in grads]),
            **{key: np.stack([g[key] for g in grads]) for key in ("dc", "drl", "dru", "dl", "du")}}


# ---- Work ----------------------------------------------------------------------------------

def _nnz(case):
    n, k = case["cols"], case["per_col"]
    if case["family"] == "blocks":
        p = case["periods"]
        return n * k + (n // p) * (p - 1)
    return n * k


def work(case):
    """The least one pass moves and computes: every matrix entry of each product with its index
    once, every vector of each step once."""
    kind, m, n, z = case["kind"], case["rows"], case["cols"], _nnz(case)
    if kind == "product":
        return {"bytes": 2 * (12 * z + 8 * (m + n)) + 4 * (m + n), "flops": 4 * z}
    # Preconditioning and norm: 11 rounds read and write the values once, 30 product pairs.
    setup_bytes = 11 * (20 * z + 16 * (m + n)) + 30 * (2 * 12 * z + 24 * (m + n))
    setup_flops = 11 * 4 * z + 30 * 4 * z
    if kind == "scaling":
        return {"bytes": setup_bytes + 8 * (z + m + n), "flops": setup_flops}
    if kind in ("call", "solve"):
        its, w = case["iterations"], 4 if case["precision"] == "mixed" else 8
        step = 2 * (w + 4) * z + 4 * (m + n) + w * (9 * n + 7 * m)
        evaluation = 2 * 12 * z + 8 * (8 * n + 8 * m)
        return {"bytes": setup_bytes + its * step + (its / 40 + 1) * evaluation,
                "flops": setup_flops + its * (6 * z + 14 * n + 14 * m) + its / 40 * 8 * z}
    if kind in ("qp", "qpcall"):
        q = n * (2 * case["band"] + 1)
        its = case["iterations"]
        step = 12 * (2 * z + q) + 8 * (8 * n + 6 * m)
        setup = 20 * (12 * (2 * z + q) + 8 * (6 * n + 2 * m))
        return {"bytes": setup + its * step,
                "flops": 20 * (4 * z + 2 * q) + its * (4 * z + 2 * q + 10 * n + 8 * m)}
    if kind == "nodes":
        # One matrix in, the nodes' vectors in and out; the iterations stay on the chip.
        c, its = case["count"], case["iterations"]
        return {"bytes": 24 * z + c * 8 * (6 * n + 4 * m),
                "flops": c * its * (6 * z + 14 * n + 14 * m) + setup_flops}
    # Backward: the LPs, points and upstream gradients in, points and gradients out; four square
    # solves of order m by conjugate gradients on a compact matrix that stays on the chip.
    c = case["count"]
    return {"bytes": c * (12 * z + 8 * (9 * n + 7 * m)), "flops": c * 4 * m * (4 * z / 2 + 10 * m)}


# ---- The same in 64 bits, by torch and numpy ------------------------------------------------

def _uniform_start(seed, count):
    """count draws of uniform_real_distribution<double>(-1, 1) over std::mt19937(seed): two
    32-bit words a draw, low word first."""
    words = np.random.RandomState(seed & 0xFFFFFFFF).randint(
        0, 1 << 32, size=2 * count, dtype=np.uint32).astype(np.float64)
    return (words[0::2] + words[1::2] * 4294967296.0) / 18446744073709551616.0 * 2.0 - 1.0


class _Sparse:
    """A and A' as torch CSR tensors in 64 bits."""

    def __init__(self, starts, index, values, m, n, device):
        self.t = torch.sparse_csr_tensor(
            torch.as_tensor(starts, dtype=torch.int64), torch.as_tensor(index, dtype=torch.int64),
            torch.as_tensor(values, dtype=torch.float64), size=(n, m)).to(device)
        cols = np.repeat(np.arange(n), np.diff(starts))
        order = np.argsort(index, kind="stable")
        rptr = np.zeros(m + 1, np.int64)
        np.cumsum(np.bincount(index, minlength=m), out=rptr[1:])
        self.a = torch.sparse_csr_tensor(
            torch.as_tensor(rptr), torch.as_tensor(cols[order], dtype=torch.int64),
            torch.as_tensor(np.asarray(values)[order], dtype=torch.float64),
            size=(m, n)).to(device)

    def mul(self, x):
        return self.a @ x

    def tmul(self, y):
        return self.t @ y


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _scale(lp):
    """Ten Ruiz rounds and one Pock-Chambolle round: (row scale, column scale, values)."""
    rows = np.asarray(lp.row_index)
    starts = np.asarray(lp.col_starts, dtype=np.int64)
    dev = _device()
    r = torch.as_tensor(rows, dtype=torch.int64, device=dev)
    c = torch.as_tensor(np.repeat(np.arange(lp.cols), np.diff(starts)), device=dev)
    v = torch.as_tensor(np.asarray(lp.values, dtype=np.float64), device=dev).clone()
    dr = torch.ones(lp.rows, dtype=torch.float64, device=dev)
    dc = torch.ones(lp.cols, dtype=torch.float64, device=dev)
    for k in range(11):
        mag = v.abs()
        how = "amax" if k < 10 else "sum"
        fr = torch.zeros_like(dr).scatter_reduce_(0, r, mag, how)
        fc = torch.zeros_like(dc).scatter_reduce_(0, c, mag, how)
        fr = torch.where(fr > 0, 1.0 / fr.sqrt(), torch.ones_like(fr))
        fc = torch.where(fc > 0, 1.0 / fc.sqrt(), torch.ones_like(fc))
        v = (v * fr[r]) * fc[c]
        dr, dc = dr * fr, dc * fc
    return dr, dc, v


def _spectral_norm(A, n, seed):
    """Thirty power steps of A'A from std::mt19937(seed + 1), with a 1% margin."""
    v = torch.as_tensor(_uniform_start(seed + 1, n), device=_device())
    norm = 0.0
    for _ in range(30):
        v = A.tmul(A.mul(v / v.norm()))
        norm = math.sqrt(float(v.norm()))
    return norm * 1.01 if norm > 0 else 1.0


def _bounds(v, absent):
    v = torch.as_tensor(np.asarray(v, dtype=np.float64), device=_device())
    return torch.where(v.abs() >= 1e30, torch.full_like(v, absent), v)


def _pdhg(lp, limit):
    """Restarted PDHG with the adaptive step in 64 bits, run to its iteration limit (no case's
    limit lets it converge): (x, reduced costs, row duals, iterations, objective)."""
    dev, inf = _device(), math.inf
    m, n = lp.rows, lp.cols
    dr, dc, vs = _scale(lp)
    raw = _Sparse(lp.col_starts, lp.row_index, lp.values, m, n, dev)
    A = _Sparse(lp.col_starts, lp.row_index, vs.cpu().numpy(), m, n, dev)
    cost = lp.sense * torch.as_tensor(lp.col_cost, device=dev)
    lo, up = _bounds(lp.col_lower, -inf), _bounds(lp.col_upper, inf)
    rl, ru = _bounds(lp.row_lower, -inf), _bounds(lp.row_upper, inf)
    c, l, u, bl, bu = cost * dc, lo / dc, up / dc, rl * dr, ru * dr
    b = torch.where(rl.isfinite(), rl, torch.where(ru.isfinite(), ru, torch.zeros_like(rl)))
    bound_norm, cost_norm = float(b.norm()), float(cost.norm())
    norm = _spectral_norm(A, n, 0)
    x = torch.zeros(n, dtype=torch.float64, device=dev).clamp(l, u)
    y = torch.zeros(m, dtype=torch.float64, device=dev)
    eta, omega = 1.0 / norm, 1.0
    ceiling = 1e3 / norm
    xs, ys, x_rst, y_rst = torch.zeros_like(x), torch.zeros_like(y), x, y
    iteration = averaged = last_restart = 0
    restart_kkt, best_kkt = inf, inf
    best = (x, y)

    def evaluate(x, y):
        ax, d = raw.mul(x), cost + raw.tmul(y)
        zero = torch.zeros_like(ax)
        primal = torch.maximum(torch.maximum(rl - ax, ax - ru), zero).norm()
        dpos, ypos = d > 0, y > 0
        side = torch.where(dpos, lo, up)
        ok = side.isfinite()
        yside = torch.where(ypos, ru, rl)
        yok = yside.isfinite()
        viol = (d[~ok] ** 2).sum() + (y[~yok] ** 2).sum()
        bc = (d[ok] * side[ok]).sum()
        support = (y[yok] * yside[yok]).sum()
        pobj, dobj = float((cost * x).sum()), float(bc - support)
        gap = abs(pobj - dobj) / (1.0 + abs(pobj) + abs(dobj))
        return max(float(primal) / (1.0 + bound_norm), float(viol.sqrt()) / (1.0 + cost_norm), gap)

    while iteration < limit:
        tau, sigma = eta / omega, eta * omega
        xn = torch.minimum(torch.maximum(x - tau * (c + A.tmul(y)), l), u)
        dx = xn - x
        adx = A.mul(dx)
        v = y + sigma * A.mul(2.0 * xn - x)
        yn = v - sigma * torch.where(bl == bu, bl, torch.minimum(torch.maximum(v / sigma, bl), bu))
        dy = yn - y
        movement = 0.5 * omega * float(dx @ dx) + 0.5 / omega * float(dy @ dy)
        interaction = abs(float(dy @ adx))
        none = interaction <= 0.0
        bar = inf if none else movement / interaction
        e = max(iteration + 1, 2)
        proposed = min((1.0 - e ** -0.3) * bar, (1.0 + e ** -0.6) * eta)
        if eta <= bar:
            x, y = xn, yn
            iteration += 1
            averaged += 1
            xs, ys = xs + x, ys + y
        if not none:
            eta = min(max(proposed, 1e-12), ceiling)
        if iteration == 0 or (iteration % 40 != 0 and not none):
            continue
        chosen = (x * dc, y * dr)
        kkt = evaluate(*chosen)
        if averaged > 0:
            mean = (xs / averaged * dc, ys / averaged * dr)
            mean_kkt = evaluate(*mean)
            if mean_kkt < kkt:
                chosen, kkt = mean, mean_kkt
        if kkt < best_kkt:
            best, best_kkt = chosen, kkt
        if kkt <= 0.2 * restart_kkt or iteration - last_restart >= max(int(0.36 * iteration), 40):
            nx, ny = float((x - x_rst).norm()), float((y - y_rst).norm())
            if nx > 1e-12 and ny > 1e-12:
                omega = math.exp(0.5 * math.log(ny / nx) + 0.5 * math.log(omega))
                omega = min(max(omega, 1e-6), 1e6)
            x_rst, y_rst, xs, ys = x, y, torch.zeros_like(x), torch.zeros_like(y)
            averaged, restart_kkt, last_restart = 0, kkt, iteration
    x, y = best
    return {"x": x, "reduced": lp.sense * (cost + raw.tmul(y)), "y": -lp.sense * y,
            "iterations": iteration,
            "objective": lp.objective_offset + float((torch.as_tensor(lp.col_cost, device=dev) * x).sum())}


def _condat_vu(qp, limit, tolerance):
    """Condat-Vu with its fixed step in 64 bits, a stopping test every 50 iterations."""
    dev, inf, lp = _device(), math.inf, qp.lp
    m, n, s = lp.rows, lp.cols, lp.sense
    A = _Sparse(lp.col_starts, lp.row_index, lp.values, m, n, dev)
    cols = np.repeat(np.arange(n), np.diff(qp.hessian_starts))
    rows, vals = np.asarray(qp.hessian_index), np.asarray(qp.hessian_values)
    off = rows != cols
    Q = torch.sparse_coo_tensor(
        torch.as_tensor(np.stack([np.concatenate([rows, cols[off]]),
                                  np.concatenate([cols, rows[off]])]), dtype=torch.int64),
        torch.as_tensor(np.concatenate([vals, vals[off]])), (n, n)).coalesce().to_sparse_csr().to(dev)
    v = torch.as_tensor(_uniform_start(26119, n), device=dev)
    norm_a = norm_q = 0.0
    if m > 0:
        for _ in range(20):
            v = A.tmul(A.mul(v / v.norm()))
            norm_a = math.sqrt(float(v.norm()))
    v = torch.as_tensor(_uniform_start(20260826, n), device=dev)
    for _ in range(20):
        v = v / v.norm()
        w = Q @ v
        norm_q, v = abs(float(v @ w)), w
    lq, a2 = 1.05 * norm_q, 1.05 ** 2 * max(norm_a ** 2, 1e-12)
    tau = 1.0 / (lq / 2.0 + math.sqrt(a2) + 1e-12)
    sigma = (1.0 / tau - lq / 2.0) / (2.0 * a2)
    c = torch.as_tensor(lp.col_cost, device=dev)
    lo, up = _bounds(lp.col_lower, -inf), _bounds(lp.col_upper, inf)
    rl, ru = _bounds(lp.row_lower, -inf), _bounds(lp.row_upper, inf)
    x = torch.zeros(n, dtype=torch.float64, device=dev).clamp(lo, up)
    y = torch.zeros(m, dtype=torch.float64, device=dev)
    t = 0
    while t < limit:
        xn = torch.minimum(torch.maximum(x - tau * (s * (c + Q @ x) + A.tmul(y)), lo), up)
        w = y + sigma * A.mul(2.0 * xn - x)
        y = w - sigma * torch.minimum(torch.maximum(w / sigma, rl), ru)
        x = xn
        t += 1
        if t % 50 == 0:
            ax = A.mul(x)
            primal = float((ax - torch.minimum(torch.maximum(ax, rl), ru)).abs().max()) if m else 0.0
            g = s * (c + Q @ x) + A.tmul(y)
            dual = float((x - torch.minimum(torch.maximum(x - g, lo), up)).abs().max())
            if primal <= tolerance and dual <= tolerance:
                break
    qx = Q @ x
    return {"x": x, "reduced": c + qx + s * A.tmul(y), "y": -s * y, "iterations": t,
            "objective": lp.objective_offset + float((c * x).sum()) + 0.5 * float((x * qx).sum())}


def _vertex_gradients(case, seed):
    """At the planted nondegenerate vertex: x*, y*, f* and the gradients by dense solves with
    the basis matrix."""
    lps, gx, gy = _backward_inputs(case, seed)
    out = {k: [] for k in ("x", "y", "f", "dc", "drl", "dru", "dl", "du")}
    dev = _device()

    def t(v):
        return torch.as_tensor(v, device=dev)

    for lp, g, h in zip(lps, gx, gy):
        cols = np.repeat(np.arange(lp.cols), np.diff(lp.col_starts))
        a = torch.zeros(lp.rows, lp.cols, dtype=torch.float64, device=dev)
        a[t(lp.row_index).long(), t(cols).long()] = t(lp.values)
        basic = t((lp.x0 > lp.col_lower) & (lp.x0 < lp.col_upper))
        x, c, zero = t(lp.x0.copy()), t(lp.col_cost), torch.zeros((), dtype=torch.float64, device=dev)
        basis = a[:, basic]
        x[basic] = torch.linalg.solve(basis, t(lp.row_lower) - a[:, ~basic] @ x[~basic])
        yp = torch.linalg.solve(basis.T, torch.stack([c[basic], t(g)[basic]], 1))
        y, p = yp[:, 0], yp[:, 1]
        dc = x.clone()
        dc[basic] += torch.linalg.solve(basis, t(h))
        d = t(g) - a.T @ p + (c - a.T @ y)
        db = p + y
        # An equality row's derivative lies on the side that its multiplier's sign names: the
        # lower side for a positive row dual.
        low, high = t(lp.x0 <= lp.col_lower), t(lp.x0 >= lp.col_upper)
        for k, v in zip(("x", "y", "f", "dc", "drl", "dru", "dl", "du"),
                        (x, y, c @ x, dc, torch.where(y > 0, db, zero),
                         torch.where(y > 0, zero, db), torch.where(~basic & low, d, zero),
                         torch.where(~basic & high, d, zero))):
            out[k].append(v)
    return {**{k: torch.stack(v) for k, v in out.items()}, "status": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("call", "solve"):
        # The mixed method's FP32 iterates have no 64-bit counterpart.
        return None if case["precision"] == "mixed" else _pdhg(_lp(case, seed), case["iterations"])
    if kind == "product":
        lp = _lp(case, seed)
        x, y = _vectors(lp, seed)
        A = _Sparse(lp.col_starts, lp.row_index, lp.values, lp.rows, lp.cols, _device())
        return {"ax": A.mul(torch.as_tensor(x, device=_device())),
                "aty": A.tmul(torch.as_tensor(y, device=_device()))}
    if kind == "scaling":
        lp = _lp(case, seed)
        dr, dc, v = _scale(lp)
        A = _Sparse(lp.col_starts, lp.row_index, v.cpu().numpy(), lp.rows, lp.cols, _device())
        return {"row_scale": dr, "col_scale": dc, "values": v,
                "norm": np.float64(_spectral_norm(A, lp.cols, 0))}
    if kind == "qp":
        return _condat_vu(_qp(case, seed), case["iterations"], 1e-9)
    if kind == "qpcall":
        return _condat_vu(_qp(case, seed), case["iterations"], 1e-8)
    if kind == "nodes":
        if case["count"] * case["iterations"] > 100 * 80:
            return None  # minutes, one node at a time
        lp = _lp(case, seed)
        got = [_pdhg(LP(lp.rows, lp.cols, lp.col_starts, lp.row_index, lp.values, lp.col_cost,
                        lo, up, lp.row_lower, lp.row_upper), case["iterations"])
               for lo, up in _node_bounds(lp, case["count"], seed)]
        return {**{k: torch.stack([g[k] for g in got]) for k in ("x", "reduced", "y")},
                "iterations": np.array([g["iterations"] for g in got]),
                "objective": np.array([g["objective"] for g in got])}
    return _vertex_gradients(case, seed)
