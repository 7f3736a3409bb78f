"""Timed cases of the PDHG engine: what a program has it do, through its public entry points.

Kinds of case (`kind`):

* ``launchers``: one iteration of the reference's driver loop and its convergence
  check through the ``sih_pdhg_launch_*`` entry points (device pointers, FP32),
  as a host program with its own loop calls them: A^T y, primal update, A x_bar,
  dual update, A x and A^T y of the new point, residuals.
* ``plain``: ``solve_gpu_pdhg``, the reference's FP32 PDHG, one whole call on host
  arrays (the call an existing caller of the reference makes).
* ``plain_resident``: the same algorithm on a ``PdhgHandle`` whose LP stays on the GPU.
* ``mixed``: ``solve_gpu_mixed``, the restarted adaptive PDHG, one whole call.
* ``mixed_resident``: the same on a ``PdhgHandle`` (``lps`` > 1: a batch), run and results read.
* ``layer``: the linear systems behind the differentiable LP layer:
  ``polish_batch`` (vertex and duals of the basis) and ``adjoint_batch`` (gradients).

``family`` says where the LP comes from: ``uniform`` (every column ``per_col``
nonzeros), ``zipf`` (column lengths Zipf(1.5) in [2, 2000]), both feasible by
construction as in ``sih_pdhg.generators``, or ``refinery`` (the multi-period
planning LP, ``periods`` blocks).  ``iterations`` is the configuration's
``max_iterations``; tolerances are the defaults (1e-4).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "refinery-optimizer_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sih_pdhg  # noqa: E402
from sih_pdhg import _lib  # noqa: E402
from sih_pdhg.generators import refinery_lp  # noqa: E402


def listed():
    return [
        # a toy LP through the launchers: seven launches, all latency
        {"name": "launchers-200x500", "kind": "launchers", "family": "uniform", "m": 200, "n": 500, "per_col": 8},
        # the differentiable layer's LP size through the launchers
        {"name": "launchers-20000x50000", "kind": "launchers", "family": "uniform", "m": 20000, "n": 50000, "per_col": 10},
        # the large skewed LP through the launchers: bandwidth and gathers
        {"name": "launchers-zipf-500000x1000000", "kind": "launchers", "family": "zipf", "m": 500000, "n": 1000000,
         "per_col": 12},
        # the call that replaces the reference's solve_pdhg, on the smallest benchmark LP with the default 4000 iterations
        {"name": "plain-2000x5000", "kind": "plain", "family": "uniform", "m": 2000, "n": 5000, "per_col": 8,
         "iterations": 4000},
        # the same algorithm on a medium skewed LP that stays on the GPU, odd sizes
        {"name": "plain-zipf-100001x199999", "kind": "plain_resident", "family": "zipf", "m": 100001, "n": 199999,
         "per_col": 12, "iterations": 1000},
        # a small LP, one whole call: set-up, copies and latency-bound steps
        {"name": "mixed-317x803", "kind": "mixed", "family": "uniform", "m": 317, "n": 803, "per_col": 7,
         "iterations": 4000},
        # the smallest benchmark LP, solved again and again while it stays on the GPU
        {"name": "mixed-2000x5000", "kind": "mixed_resident", "family": "uniform", "m": 2000, "n": 5000, "per_col": 8,
         "lps": 1, "iterations": 4000},
        # refinery planning, one day in hourly periods
        {"name": "mixed-refinery-24", "kind": "mixed_resident", "family": "refinery", "periods": 24, "lps": 1,
         "iterations": 2048},
        # refinery planning, one week in hourly periods
        {"name": "mixed-refinery-168", "kind": "mixed_resident", "family": "refinery", "periods": 168, "lps": 1,
         "iterations": 2048},
        # the large skewed LP of the benchmark's default workload
        {"name": "mixed-zipf-500000x1000000", "kind": "mixed_resident", "family": "zipf", "m": 500000, "n": 1000000,
         "per_col": 12, "lps": 1, "iterations": 1024},
        # a batch of independent scenarios solved together
        {"name": "mixed-batch-64x2000x5000", "kind": "mixed_resident", "family": "uniform", "m": 2000, "n": 5000,
         "per_col": 8, "lps": 64, "iterations": 1024},
        # forward polish and backward of a layer of 16 small LPs
        {"name": "layer-16x200x500", "kind": "layer", "m": 200, "n": 500, "per_col": 8, "lps": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["launchers", "plain", "plain_resident", "mixed", "mixed_resident", "mixed_resident", "batch",
                       "layer"])
    if kind == "layer":
        return {"kind": kind, "m": _log(rng, 40, 200), "n": _log(rng, 500, 700), "per_col": rng.randint(4, 9),
                "lps": rng.randint(1, 16)}
    if kind == "mixed_resident" and rng.random() < 0.5:
        return {"kind": kind, "family": "refinery", "periods": _log(rng, 6, 168), "lps": 1,
                "iterations": _log(rng, 256, 2048)}
    lps = _log(rng, 2, 64) if kind == "batch" else 1
    top = {"launchers": 500000, "plain": 20000, "plain_resident": 100000, "mixed": 20000, "mixed_resident": 500000,
           "batch": 2000}[kind]
    m = _log(rng, 200, top)
    c = {"kind": "mixed_resident" if kind == "batch" else kind, "family": rng.choice(["uniform", "zipf"]), "m": m,
         "n": int(m * rng.uniform(1.5, 2.5)), "per_col": rng.randint(5, 12)}
    if c["kind"] == "mixed_resident":
        c["lps"] = lps
    if kind != "launchers":
        c["iterations"] = _log(rng, 256, 1024)
    return c


# ---------------------------------------------------------------------------- inputs
def _random_lp(case, seed):
    """A feasible, bounded random LP, drawn on the GPU (the recipe of
    sih_pdhg.generators.random_feasible_lp): FP64 tensors and int64 indices."""
    m, n, per_col = case["m"], case["n"], case["per_col"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    d = dict(device="cuda", dtype=torch.float64)
    rand = lambda k: torch.rand(k, generator=g, **d)  # noqa: E731
    if case["family"] == "uniform":
        counts = torch.full((n,), min(per_col, m), device="cuda", dtype=torch.int64)
    else:  # Zipf(1.5): P(X > x) ~ x^-1/2, clipped to [2, 2000], rescaled to per_col on the mean
        raw = rand(n).clamp_min(1e-12).pow(-2.0).floor().clamp(2, 2000)
        counts = (raw * (per_col * n / raw.sum()) + rand(n)).floor().clamp(2, min(2000, m)).to(torch.int64)
    cols = torch.repeat_interleave(torch.arange(n, device="cuda"), counts)
    rows = torch.randint(0, m, (cols.numel(),), generator=g, device="cuda")
    key = torch.unique(cols * m + rows)  # sorted by column, then row; a row drawn twice in a column counts once
    cols, rows = key // m, key % m
    vals = torch.randn(key.numel(), generator=g, **d)
    upper = 1.0 + 9.0 * rand(n)
    x0 = upper * rand(n)
    y0 = torch.randn(m, generator=g, **d)
    meq = m // 2
    y0[meq:] = -y0[meq:].abs()
    cp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    cp[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
    order = torch.argsort(rows * n + cols)
    rp = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    # host sums: index_add_ and cumsum on the GPU add in no fixed order
    ax0 = torch.from_numpy(np.bincount(rows.cpu().numpy(), weights=(vals * x0[cols]).cpu().numpy(), minlength=m)).cuda()
    c = torch.from_numpy(np.bincount(cols.cpu().numpy(), weights=(vals * y0[rows]).cpu().numpy(), minlength=n)).cuda()
    c += rand(n)
    slack = rand(m)
    lo, hi = ax0.clone(), ax0.clone()
    lo[meq:] = -math.inf
    hi[meq:] += slack[meq:]
    return {"m": m, "n": n, "cp": cp, "ri": rows, "cv": vals, "rp": rp, "ci": cols[order], "rv": vals[order], "c": c,
            "l": torch.zeros_like(c), "u": upper, "rl": lo, "ru": hi}


def _problem(case, seed):
    if case["family"] == "refinery":
        # one plant (data seed 0) under another price scenario each time, as the scenario batches draw them
        r = np.random.default_rng(seed)
        p = refinery_lp(case["periods"], 0, r.lognormal(0.0, 0.15, 3), r.lognormal(0.0, 0.15, 145))
        p.A.csr_values()
        return p
    a = {k: (v.cpu().numpy() if torch.is_tensor(v) else v) for k, v in _random_lp(case, seed).items()}
    A = sih_pdhg.SparseMatrix(a["m"], a["n"], a["cp"], a["ri"], a["cv"], a["rp"], a["ci"], a["rv"])
    return sih_pdhg.Problem.from_arrays(A, a["c"], a["l"], a["u"], a["rl"], a["ru"])


def _layer_lp(case, seed):
    """A small LP with a known vertex solution: the first k columns basic, the
    equality rows and half of the inequality rows active, B = A[active, basic]
    with one large entry per row (a matching), so that it is well conditioned."""
    m, n, per_col = case["m"], case["n"], case["per_col"]
    r = np.random.default_rng(seed)
    meq = m // 2
    k = meq + (m - meq + 1) // 2  # active rows [0, k) = basic columns [0, k)
    rows = np.argsort(r.random((n, m)), axis=1)[:, :per_col]
    vals = r.standard_normal((n, per_col))
    dense = np.zeros((m, n))
    dense[rows.T, np.arange(n)] = vals.T
    dense[np.arange(k), r.permutation(k)] += np.where(r.random(k) < 0.5, -6.0, 6.0)
    col, row = np.nonzero(dense.T)
    cp = np.concatenate([[0], np.cumsum(np.bincount(col, minlength=n))])
    upper = r.uniform(1.0, 10.0, n)
    x = np.where(r.random(n) < 0.5, 0.0, upper)
    x[:k] = r.uniform(0.2, 0.8, k) * upper[:k]
    y = np.zeros(m)  # simplex duals
    y[:k] = r.standard_normal(k)
    y[meq:k] = -np.abs(y[meq:k])
    y[:k] += np.where(y[:k] < 0, -0.1, 0.1)
    red = np.where(x == 0.0, 1.0, -1.0) * r.uniform(0.2, 1.0, n)
    red[:k] = 0.0
    ax = dense @ x
    lo, hi = ax.copy(), ax.copy()
    lo[meq:] = -np.inf
    hi[k:] += r.uniform(0.5, 1.0, m - k)
    A = sih_pdhg.SparseMatrix(m, n, cp, row, dense[row, col])
    p = sih_pdhg.Problem.from_arrays(A, dense.T @ y + red, np.zeros(n), upper, lo, hi)
    # what a solve returns: the point to a few digits, row duals in the PDHG sign
    return {"p": p, "dense": dense, "k": k, "x": x * (1.0 + 1e-5 * r.standard_normal(n)), "x_exact": x,
            "y": -y * (1.0 + 1e-5 * r.standard_normal(m)), "y_exact": -y, "g": r.standard_normal(n)}


def _f32(a):
    return a.to(torch.float32).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "launchers":
        a = _random_lp(case, seed)
        i32 = lambda v: v.to(torch.int32).contiguous()  # noqa: E731
        t = {k: i32(a[k]) for k in ("cp", "ri", "rp", "ci")}
        t.update({k: _f32(a[k]) for k in ("cv", "rv", "c", "l", "u", "rl", "ru")})
        m, n = a["m"], a["n"]
        # step sizes 0.95 / max(1, sum |a|) as the reference's driver sets them, start x = 0, a dual some way off zero
        def step(ptr, vals):
            at = np.repeat(np.arange(ptr.numel() - 1), np.diff(ptr.cpu().numpy()))
            sums = np.bincount(at, weights=vals.abs().cpu().numpy(), minlength=ptr.numel() - 1)
            return _f32(torch.from_numpy(0.95 / np.maximum(sums, 1.0)).cuda())

        t["tau"], t["sigma"] = step(a["cp"], a["cv"]), step(a["rp"], a["rv"])
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        t["x"] = _f32(a["u"] * torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
        t["xbar"] = t["x"].clone()
        t["y"] = 0.1 * torch.randn(m, generator=g, device="cuda")
        for k, size in (("aty", n), ("axbar", m), ("ax", m), ("aty2", n), ("rowv", m), ("colv", n)):
            t[k] = torch.zeros(size, device="cuda")
        p = {k: v.data_ptr() for k, v in t.items()}
        s = torch.cuda.current_stream().cuda_stream
        lib = _lib.load()
        torch.cuda.synchronize()
        calls = [
            (lib.sih_pdhg_launch_csc_spmv, (n, p["cp"], p["ri"], p["cv"], p["y"], p["aty"], s)),
            (lib.sih_pdhg_launch_primal_update, (n, p["tau"], p["c"], p["aty"], p["l"], p["u"], p["x"], p["xbar"], s)),
            (lib.sih_pdhg_launch_csr_spmv, (m, p["rp"], p["ci"], p["rv"], p["xbar"], p["axbar"], s)),
            (lib.sih_pdhg_launch_dual_update, (m, p["sigma"], p["axbar"], p["rl"], p["ru"], p["y"], s)),
            (lib.sih_pdhg_launch_csr_spmv, (m, p["rp"], p["ci"], p["rv"], p["x"], p["ax"], s)),
            (lib.sih_pdhg_launch_csc_spmv, (n, p["cp"], p["ri"], p["cv"], p["y"], p["aty2"], s)),
            (lib.sih_pdhg_launch_residuals, (m, n, p["ax"], p["rl"], p["ru"], p["rowv"], p["x"], p["c"], p["aty2"],
                                             p["l"], p["u"], p["tau"], p["colv"], s)),
        ]
        return {"kind": kind, "t": t, "calls": calls}
    if kind == "layer":
        lps = [_layer_lp(case, 1000 * seed + b) for b in range(case["lps"])]
        return {"kind": kind, "ps": [q["p"] for q in lps], "xs": [q["x"] for q in lps], "ys": [q["y"] for q in lps],
                "gs": [q["g"] for q in lps]}
    cfg = sih_pdhg.GpuPdhgConfig(max_iterations=case["iterations"])
    if kind in ("plain", "mixed"):
        return {"kind": kind, "p": _problem(case, seed), "cfg": cfg}
    ps = [_problem(case, 1000 * seed + b) for b in range(case.get("lps", 1))]
    # autotune=0: the tuner's choice (by timing) fixes the order of the sums, so that a run with it on is not repeatable
    h = sih_pdhg.PdhgHandle(ps, cfg, autotune=0,
                            algorithm=sih_pdhg.ALGO_PLAIN if kind == "plain_resident" else sih_pdhg.ALGO_MIXED)
    return {"kind": kind, "h": h, "lps": len(ps)}


# ---------------------------------------------------------------------------- one pass
def _outputs(sols):
    cat = lambda k: np.concatenate([getattr(s, k) for s in sols])  # noqa: E731
    return {"x": cat("x"), "row_duals": cat("row_duals"), "slack": cat("slack"), "reduced_costs": cat("reduced_costs"),
            "objective": np.array([s.primal_objective for s in sols]),
            "iterations": np.array([s.simplex_iterations for s in sols]),
            "status": np.array([int(s.status) for s in sols])}


def run(state):
    kind = state["kind"]
    if kind == "launchers":
        for fn, args in state["calls"]:
            _lib.check(fn(*args))
        t = state["t"]
        return {k: t[k] for k in ("x", "xbar", "y", "ax", "aty2", "rowv", "colv")}
    if kind == "plain":
        return _outputs([sih_pdhg.solve_gpu_pdhg(state["p"], state["cfg"])])
    if kind == "mixed":
        return _outputs([sih_pdhg.solve_gpu_mixed(state["p"], state["cfg"])])
    if kind == "layer":
        xs, ys, _ = sih_pdhg.polish_batch(state["ps"], state["xs"], state["ys"])
        grads, _ = sih_pdhg.adjoint_batch(state["ps"], xs, ys, state["gs"])
        cat = lambda k: np.concatenate([g[k] for g in grads])  # noqa: E731
        return {"x": np.concatenate(xs), "row_duals": np.concatenate(ys),
                **{k: cat(k) for k in ("row_lower", "row_upper", "col_lower", "col_upper")}}
    state["h"].run()
    return _outputs([state["h"].result(b) for b in range(state["lps"])])


# ---------------------------------------------------------------------------- floors
def _sizes(case):
    if case.get("family") == "refinery":  # per period of the plant with data seed 0
        return 892 * case["periods"], 1414 * case["periods"], 6527 * case["periods"]
    return case["m"], case["n"], case["n"] * case["per_col"]


def work(case):
    """Bytes and operations of one pass: per step, the matrix once in each
    direction (index and value, 8 bytes a nonzero) and the vectors of the
    updates once; 2 operations per nonzero and direction."""
    m, n, nnz = _sizes(case)
    kind = case["kind"]
    if kind == "launchers":  # two products of each kind; the updates' and the residuals' vectors
        return {"bytes": 4 * 8 * nnz + 4 * (16 * n + 13 * m), "flops": 8 * nnz}
    if kind == "layer":  # three systems of about 100 CGLS steps
        steps = 300
        return {"bytes": case["lps"] * steps * (16 * nnz + 4 * (6 * n + 6 * m)), "flops": case["lps"] * steps * 4 * nnz}
    # random LPs reach 1e-4 after about 1,000 steps of the adaptive algorithm
    steps = case["iterations"] if kind.startswith("plain") else min(case["iterations"], 1024)
    if case.get("family") == "refinery":
        steps = case["iterations"]
    lps = case.get("lps", 1)
    return {"bytes": lps * steps * (16 * nnz + 4 * (10 * n + 8 * m)), "flops": lps * steps * 4 * nnz}


# ---------------------------------------------------------------------------- 64-bit values
def _exact_launchers(case, seed):
    t = prepare(case, seed)["t"]
    d = {k: (v.double() if v.is_floating_point() else v.long()) for k, v in t.items()}
    col = torch.repeat_interleave(torch.arange(case["n"], device="cuda"), torch.diff(d["cp"]))
    row = torch.repeat_interleave(torch.arange(case["m"], device="cuda"), torch.diff(d["rp"]))
    at = lambda y: torch.zeros_like(d["c"]).index_add_(0, col, d["cv"] * y[d["ri"]])  # noqa: E731
    ax = lambda x: torch.zeros_like(d["sigma"]).index_add_(0, row, d["rv"] * x[d["ci"]])  # noqa: E731
    x = torch.minimum(torch.maximum(d["x"] - d["tau"] * (d["c"] + at(d["y"])), d["l"]), d["u"])
    xbar = 2.0 * x - d["x"]
    w = ax(xbar) + d["y"] / d["sigma"]
    y = d["sigma"] * (w - torch.minimum(torch.maximum(w, d["rl"]), d["ru"]))
    axn, atn = ax(x), at(y)
    rowv = torch.maximum(torch.relu(d["rl"] - axn), torch.relu(axn - d["ru"]))
    proj = torch.minimum(torch.maximum(x - d["tau"] * (d["c"] + atn), d["l"]), d["u"])
    return {"x": x, "xbar": xbar, "y": y, "ax": axn, "aty2": atn, "rowv": rowv,
            "colv": (x - proj).abs() / d["tau"].clamp_min(1e-4)}


def _exact_plain(case, seed):
    """The reference's PDHG in 64 bits (dense-free, on the GPU): best checked point and last dual."""
    a = _random_lp(case, seed)
    m, n = a["m"], a["n"]
    At = torch.sparse_csr_tensor(a["cp"], a["ri"], a["cv"], size=(n, m))
    A = torch.sparse_csr_tensor(a["rp"], a["ci"], a["rv"], size=(m, n))
    row = torch.repeat_interleave(torch.arange(m, device="cuda"), torch.diff(a["rp"]))
    col = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.diff(a["cp"]))
    sigma = 0.95 / torch.zeros(m, device="cuda", dtype=torch.float64).index_add_(0, row, a["rv"].abs()).clamp_min(1.0)
    tau = 0.95 / torch.zeros(n, device="cuda", dtype=torch.float64).index_add_(0, col, a["cv"].abs()).clamp_min(1.0)
    b = torch.cat([a["rl"][torch.isfinite(a["rl"])], a["ru"][torch.isfinite(a["ru"])]]).abs().max().clamp_min(1.0)
    cm = a["c"].abs().max().clamp_min(1.0)
    x, y = torch.zeros_like(a["c"]), torch.zeros_like(a["rl"])
    clip = lambda v, lo, hi: torch.minimum(torch.maximum(v, lo), hi)  # noqa: E731
    best, best_x, it = torch.tensor(1e30, device="cuda", dtype=torch.float64), x.clone(), 0
    for it in range(1, case["iterations"] + 1):
        xn = clip(x - tau * (a["c"] + At @ y), a["l"], a["u"])
        w = A @ (2.0 * xn - x) + y / sigma
        y = sigma * (w - clip(w, a["rl"], a["ru"]))
        x = xn
        if it % 25 == 0 or it == case["iterations"]:
            axn = A @ x
            p = torch.maximum(torch.relu(a["rl"] - axn), torch.relu(axn - a["ru"])).max() / b
            proj = clip(x - tau * (a["c"] + At @ y), a["l"], a["u"])
            q = ((x - proj).abs() / tau.clamp_min(1e-4)).max() / cm
            if torch.maximum(p, q) < best:
                best, best_x = torch.maximum(p, q), x.clone()
            if p <= 1e-4 and q <= 1e-4:
                break
    return {"x": best_x, "row_duals": y, "slack": A @ best_x, "reduced_costs": a["c"] + At @ y,
            "objective": (a["c"] @ best_x).reshape(1), "iterations": None, "status": None}


def _exact_layer(case, seed):
    out = {k: [] for k in ("x", "row_duals", "row_lower", "row_upper", "col_lower", "col_upper")}
    for b in range(case["lps"]):
        q = _layer_lp(case, 1000 * seed + b)
        k, A, g, m, n = q["k"], q["dense"], q["g"], case["m"], case["n"]
        lam = np.zeros(m)
        lam[:k] = np.linalg.solve(A[:k, :k].T, g[:k])
        gj = g - A.T @ lam
        gj[:k] = 0.0
        low = q["x_exact"] == 0.0
        out["x"].append(q["x_exact"])
        out["row_duals"].append(q["y_exact"])
        eq = np.arange(m) < m // 2
        out["row_lower"].append(np.where(eq, lam, 0.0))
        out["row_upper"].append(np.where(eq, 0.0, lam))
        out["col_lower"].append(np.where(low, gj, 0.0))
        out["col_upper"].append(np.where(low, 0.0, gj))
    return {k: np.concatenate(v) for k, v in out.items()}


def exact(case, seed):
    """64-bit values of run()'s outputs.  None for the adaptive algorithm: its
    step sizes and restarts follow its own rounding, so that the point it stops
    at has no value of its own."""
    kind = case["kind"]
    if kind == "launchers":
        return _exact_launchers(case, seed)
    if kind == "layer":
        return _exact_layer(case, seed)
    if kind == "plain" or kind == "plain_resident":
        return _exact_plain(case, seed if kind == "plain" else 1000 * seed)
    return None
