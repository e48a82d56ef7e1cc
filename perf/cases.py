"""Timed cases of the engine: the calls a program makes, over the range of
sizes, precisions and directions it makes them in.

  solve     one LP through Problem.solve (a kept handle) or solve_lp (host
            arrays in, answer out), a fixed budget of PDHG iterations
  batch     solve_batch: many small LPs in one call, to a tolerance
  layer     the differentiable LP layer: inference, or a training step with
            the gradients of every input
  evaluate  KKT metrics of a point held in device memory, through the
            allocation-free entry point

listed() names the cases, draw(rng) gives others of the same ranges.
"""
import ctypes as C
import math
import types

import numpy as np
import torch

from igaos_gb300 import capi, generators
from igaos_gb300.layer import BatchPattern, stack_lps, unrolled_lp


def listed():
    return [
        # a control loop or a unit test: one tiny LP from host arrays, where
        # setup and launch latency are all there is
        dict(name="solve_tiny", kind="solve", shape="random", m=60, n=150, nnz=450, handle=False,
             precision="fp64", iterations=1024),
        # the small random LP of the benchmark (2,000 x 5,000), re-solved on a
        # kept handle in FP32 + refinement
        dict(name="solve_small", kind="solve", shape="random", m=2000, n=5000, nnz=20000,
             handle=True, precision="fp32-refine", iterations=2048),
        # one call on a mid-size LP with Zipf column lengths (20,000 x 50,000,
        # the size of the golden optimum): upload, scaling, solve, free
        dict(name="solve_medium", kind="solve", shape="zipf", m=20000, n=50000, nnz=500000,
             handle=False, precision="fp32-refine", iterations=1024),
        # the large sparse LP of the benchmark in the default precision
        dict(name="solve_large", kind="solve", shape="zipf", m=200000, n=500000, nnz=5000000,
             handle=True, precision="fp64", iterations=256),
        # multicommodity flow on the benchmark's 300 x 300 grid (8.6 million
        # nonzeros, columns of three entries)
        dict(name="solve_flow", kind="solve", shape="flow", side=300, commodities=8, handle=True,
             precision="fp32-refine", iterations=256),
        # many small planning problems at once
        dict(name="batch_small", kind="batch", count=512, m_lo=20, m_hi=120, tolerance=1e-6),
        # the uneven batch of the benchmark, one wave of it
        dict(name="batch_uneven", kind="batch", count=160, m_lo=20, m_hi=800, tolerance=1e-4),
        # inference through the layer: a few ragged small LPs, forward only
        dict(name="layer_infer", kind="layer", dtype="float32", count=16, m_lo=12, m_hi=60, ratio=2.0,
             density=0.1, iterations=200, checkpoint=50, backward=False),
        # the training step of the benchmark: 256 LPs of 500 x 1,000
        dict(name="layer_train", kind="layer", dtype="float32", count=256, m_lo=500, m_hi=500,
             ratio=2.0, density=0.02, iterations=1000, checkpoint=50, backward=True),
        # the same layer in double precision (gradient checks, ill-scaled LPs)
        dict(name="layer_train_f64", kind="layer", dtype="float64", count=96, m_lo=500, m_hi=500,
             ratio=2.0, density=0.02, iterations=200, checkpoint=50, backward=True),
        # a training step on a ragged batch whose largest LPs do not fit on chip
        dict(name="layer_ragged", kind="layer", dtype="float32", count=96, m_lo=40, m_hi=1300,
             ratio=2.0, density=0.02, iterations=200, checkpoint=32, backward=True),
        # checking a point of the large LP from a program that owns its memory
        dict(name="evaluate", kind="evaluate", shape="zipf", m=200000, n=500000, nnz=5000000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "layer", "layer", "evaluate"])
    if kind in ("solve", "evaluate"):
        shape = rng.choice(["random", "zipf", "flow"])
        if shape == "flow":
            case = dict(kind=kind, shape=shape, side=_log(rng, 8, 250), commodities=rng.randint(2, 8))
            size = case["side"] ** 2 * case["commodities"] * 12
        else:
            m = _log(rng, 40, 150000)
            n = int(m * rng.uniform(1.2, 3.5))
            case = dict(kind=kind, shape=shape, m=m, n=n, nnz=int(n * rng.uniform(2.5, 9.0)))
            size = case["nnz"]
        if kind == "solve":
            case["handle"] = rng.random() < 0.5
            case["precision"] = rng.choice(["fp64", "fp32-refine"])
            case["iterations"] = max(64, min(2048, int(2e8 / max(size, 1)) // 64 * 64))
        return case
    if kind == "batch":
        m_hi = _log(rng, 60, 600)
        return dict(kind=kind, count=_log(rng, 24, 256), m_lo=rng.randint(12, 40), m_hi=m_hi,
                    tolerance=rng.choice([1e-4, 1e-4, 1e-6]) if m_hi < 150 else 1e-4)
    m_hi = _log(rng, 30, 1200)
    dtype = rng.choice(["float32", "float64"])
    if dtype == "float64":
        m_hi = min(m_hi, 700)
    density = min(0.2, rng.uniform(8.0, 24.0) / m_hi)
    return dict(kind=kind, dtype=dtype, count=_log(rng, 8, 160), m_lo=max(8, int(m_hi * rng.uniform(0.1, 1.0))),
                m_hi=m_hi, ratio=round(rng.uniform(1.3, 2.5), 2), density=round(density, 4),
                iterations=rng.randint(60, 300), checkpoint=rng.choice([10, 25, 50, 64]),
                backward=rng.random() < 0.7)


# ---------------------------------------------------------------- inputs
def _sparse_lp(shape, m, n, nnz, seed):
    """The random and Zipf shapes of generators.random_lp / config2, with the
    index sorting on the GPU (those take seconds in numpy at full size)."""
    rng = np.random.default_rng(seed)
    if shape == "random":
        rows = np.concatenate([rng.integers(0, m, n), rng.integers(0, m, max(0, nnz - n))])
        cols = np.concatenate([np.arange(n), rng.integers(0, n, max(0, nnz - n))])
    else:
        deg = np.minimum(rng.zipf(1.5, n), 2000).astype(np.float64)
        deg = np.minimum(np.maximum(1, np.rint(deg * (nnz / deg.sum()))), m).astype(np.int64)
        cols = np.repeat(np.arange(n), deg)
        rows = rng.integers(0, m, cols.shape[0])
    key = torch.unique(torch.from_numpy(cols * m + rows).cuda())  # sorted: column, then row
    cols, rows = key // m, key % m
    order = torch.sort(rows, stable=True).indices
    point = lambda v, k: torch.cumsum(torch.bincount(v + 1, minlength=k + 1), 0).int().cpu().numpy()
    k = key.shape[0]
    if shape == "random":
        acx = rng.standard_normal(k)
    else:
        acx = 10.0 ** rng.uniform(-3.0, 3.0, k) * rng.choice([-1.0, 1.0], k)
    order_h, rows_h, cols_h = order.cpu().numpy(), rows.cpu().numpy(), cols.cpu().numpy()
    xs = rng.uniform(0.0, 10.0, n)
    ax_star = np.bincount(rows_h, weights=acx * xs[cols_h], minlength=m)
    rmin, rmax = generators._feasible_rows(rng, None, ax_star, m // 2)
    return generators.LPData(
        m=m, n=n, ap=point(rows, m), ai=cols_h[order_h].astype(np.int32), ax=acx[order_h],
        cp=point(cols, n), ci=rows_h.astype(np.int32), acx=acx, c=rng.standard_normal(n),
        cl=np.zeros(n), cu=np.full(n, 10.0), rmin=rmin, rmax=rmax, meta=dict(x_star=xs))


def _lp(case, seed):
    if case["shape"] == "flow":
        return generators.config5(seed, side=case["side"], commodities=case["commodities"])
    return _sparse_lp(case["shape"], case["m"], case["n"], case["nnz"], seed)


def _small_lps(case, seed):
    """The LPs of a batch. Their sizes belong to the case, not to the seed; a
    layer's sparsity pattern too (a program builds its BatchPattern once and
    feeds it new values)."""
    fixed = np.random.default_rng([case["count"], case["m_lo"], case["m_hi"]])
    rng = np.random.default_rng(seed)
    lo, hi = math.log(case["m_lo"]), math.log(max(case["m_lo"], case["m_hi"]))
    ratio, density = case.get("ratio", 2.5), case.get("density", 0.01)
    out = []
    for _ in range(case["count"]):
        m = int(round(math.exp(fixed.uniform(lo, hi))))
        n = max(2, int(round(ratio * m)))
        if case["kind"] == "batch":
            out.append(generators.bernoulli_lp(rng, m, n, density, 5.0))
            continue
        lp = generators.bernoulli_lp(fixed, m, n, density, 10.0)
        rows = np.repeat(np.arange(m), np.diff(lp.ap))
        lp.ax = rng.standard_normal(lp.ax.shape[0])
        lp.c = rng.standard_normal(n)
        ax_star = np.bincount(rows, weights=lp.ax * rng.uniform(0.0, 10.0, n)[lp.ai], minlength=m)
        lp.rmin, lp.rmax = generators._feasible_rows(rng, None, ax_star, m // 2)
        out.append(lp)
    return out


def _point(lp, seed):
    """A point as a solver's later iterations give: near x*, some columns at
    a bound, duals whose sign each row's finite bound allows."""
    rng = np.random.default_rng(seed + 1)
    x = lp.meta["x_star"] if "x_star" in lp.meta else rng.uniform(0.0, 1.0, lp.n) * lp.cu
    x = np.clip(x + 1e-3 * rng.standard_normal(lp.n), lp.cl, lp.cu)
    x = np.where(rng.random(lp.n) < 0.3, lp.cl, x)
    y = rng.standard_normal(lp.m) * (rng.random(lp.m) < 0.6)
    return x, np.where((y > 0) & ~np.isfinite(lp.rmax) | (y < 0) & ~np.isfinite(lp.rmin), 0.0, y)


_VALUES = ("ax", "acx", "c", "cl", "cu", "rmin", "rmax")
_INDEX = ("ap", "ai", "cp", "ci")
_ENTRY = ("ap", "ai", "ax", "cp", "ci", "acx", "c", "cl", "cu", "rmin", "rmax", "x", "y", "out")


def prepare(case, seed):
    s = types.SimpleNamespace(case=case)
    if case["kind"] == "solve":
        s.lp = _lp(case, seed)
        s.opts = dict(precision=case["precision"], tolerance=1e-8, time_limit=1e9,
                      max_iterations=case["iterations"])
        s.problem = capi.Problem(s.lp) if case["handle"] else None
    elif case["kind"] == "batch":
        s.lps = _small_lps(case, seed)
    elif case["kind"] == "layer":
        lps = _small_lps(case, seed)
        dtype = getattr(torch, case["dtype"])
        s.pattern = BatchPattern.from_lps(lps, "cuda")
        s.data = [t.requires_grad_(case["backward"]) for t in stack_lps(lps, dtype, "cuda")]
        if case["backward"]:  # the loss weighs x and the objective
            g = torch.Generator().manual_seed(seed)
            s.wx = torch.randn(s.pattern.total_n, generator=g, dtype=dtype).cuda()
            s.wo = torch.rand(s.pattern.count, generator=g, dtype=dtype).cuda()
    else:
        lp = _lp(case, seed)
        x, y = _point(lp, seed)
        s.m, s.n = lp.m, lp.n
        s.t = {k: torch.from_numpy(np.ascontiguousarray(getattr(lp, k), np.float64)).cuda()
               for k in _VALUES}
        s.t.update({k: torch.from_numpy(np.ascontiguousarray(getattr(lp, k), np.int32)).cuda()
                    for k in _INDEX})
        s.t.update(x=torch.from_numpy(x).cuda(), y=torch.from_numpy(y).cuda(),
                   out=torch.zeros(6, dtype=torch.float64, device="cuda"))
    return s


# ------------------------------------------------------------------ a pass
def run(s):
    case = s.case
    if case["kind"] == "solve":
        r = s.problem.solve(**s.opts) if s.problem else capi.solve_lp(s.lp, **s.opts)
        return {k: r[k] for k in ("x", "y", "objective", "iterations", "status")}
    if case["kind"] == "batch":
        out = capi.solve_batch(s.lps, tolerance=case["tolerance"], max_iterations=200000)
        return {"x": np.concatenate([r["x"] for r in out]), "y": np.concatenate([r["y"] for r in out]),
                "objective": np.array([r["objective"] for r in out]),
                "iterations": np.array([r["iterations"] for r in out]),
                "status": np.array([r["status"] for r in out])}
    if case["kind"] == "layer":
        x, y, obj = unrolled_lp(s.pattern, *s.data, iterations=case["iterations"],
                                checkpoint=case["checkpoint"])
        res = {"x": x, "y": y, "obj": obj}
        if case["backward"]:
            loss = (s.wx * x).sum() + (s.wo * obj).sum()
            grads = torch.autograd.grad(loss, s.data)
            res.update(zip(("gc", "gcl", "gcu", "grmin", "grmax", "gax"), grads))
        return res
    stream = torch.cuda.current_stream().cuda_stream
    capi._check(capi.lib().igaos_pdhg_evaluate_noalloc(
        s.m, s.n, *[C.c_void_p(s.t[k].data_ptr()) for k in _ENTRY], C.c_void_p(stream)))
    return {"metrics": s.t["out"]}


# ----------------------------------------------------------------- counts
def work(case):
    """Every input read once, every answer written once, and the operations
    of the iterations (a product A x or A^T y is two per nonzero)."""
    if case["kind"] in ("solve", "evaluate"):
        if case["shape"] == "flow":
            arcs = 4 * case["side"] * (case["side"] - 1)
            n = arcs * case["commodities"]
            m = case["side"] ** 2 * case["commodities"] + arcs
            nnz = 3 * n
        else:
            m, n, nnz = case["m"], case["n"], case["nnz"]
        size = nnz * 2 * 12 + (m + n) * (4 + 8 * 4)
        if case["kind"] == "evaluate":
            return {"bytes": size, "flops": 4 * nnz}
        return {"bytes": size, "flops": case["iterations"] * (4 * nnz + 20 * (m + n))}
    a, b = math.log(case["m_lo"]), math.log(max(case["m_lo"], case["m_hi"]))
    mean = lambda p: math.exp(a * p) if b <= a else (math.exp(b * p) - math.exp(a * p)) / (p * (b - a))
    ratio, density = case.get("ratio", 2.5), case.get("density", 0.01)
    m = case["count"] * mean(1)
    n = m * ratio
    nnz = case["count"] * ratio * density * mean(2)
    if case["kind"] == "batch":  # a few hundred iterations at the least
        return {"bytes": 12 * nnz + 40 * (m + n), "flops": 500 * (4 * nnz + 20 * (m + n))}
    es = 8 if case["dtype"] == "float64" else 4
    products = case["iterations"] * (4 if case["backward"] else 2) + 200
    factor = 2 if case["backward"] else 1
    return {"bytes": factor * (es + 12) * nnz + factor * 5 * es * (m + n),
            "flops": products * 2 * nnz + case["iterations"] * 12 * (m + n)}


# ------------------------------------------------ the same in plain 64 bits
def exact(case, seed):
    if case["kind"] == "evaluate":
        return _exact_evaluate(case, seed)
    if case["kind"] == "layer":
        return _exact_layer(case, seed)
    # a budget of adaptive iterations has no value of its own in exact
    # arithmetic (the step sizes and restarts follow the rounding)
    return None


def _exact_evaluate(case, seed):
    lp = _lp(case, seed)
    x, y = _point(lp, seed)
    rows = np.repeat(np.arange(lp.m), np.diff(lp.ap))
    ax = np.bincount(rows, weights=lp.ax * x[lp.ai], minlength=lp.m)
    d = lp.c + np.bincount(lp.ai, weights=lp.ax * y[rows], minlength=lp.n)
    viol = np.maximum(lp.rmin - ax, ax - lp.rmax)
    pinf = max(0.0, viol.max()) / (1.0 + np.abs(np.clip(ax, lp.rmin, lp.rmax)).max())
    fin = lambda v: np.where(np.isfinite(v), np.abs(v), 0.0)
    scale = np.maximum(np.abs(ax), np.maximum(fin(lp.rmin), fin(lp.rmax)))
    prow = (np.maximum(0.0, viol) / (1.0 + scale)).max()
    tol = 1e-9 * (1.0 + np.abs(np.where(np.isfinite(lp.cu), lp.cu, lp.cl)))
    free = ~((x <= lp.cl + tol) & (d > 0) | (x >= lp.cu - tol) & (d < 0))
    cmax = np.abs(lp.c).max()
    dinf = np.abs(d[free]).max(initial=0.0) / (1.0 + cmax)
    op = float(lp.c @ x)
    side = np.where(d >= 0, lp.cl, lp.cu)
    yz = 1e-8 * (1.0 + np.abs(y).max())
    rside = np.where(y > yz, lp.rmax, np.where(y < -yz, lp.rmin, 0.0))
    od = float(np.sum(d * side) - np.sum(np.where(np.abs(y) > yz, y, 0.0) * rside))
    gap = max(0.0, op - od) / (1.0 + abs(op))
    return {"metrics": np.array([pinf, dinf, gap, op, od, prow])}


def _exact_layer(case, seed):
    """The unrolled iteration on dense matrices, instances of a like size in
    one batch, with torch's reverse mode for the gradients."""
    lps = _small_lps(case, seed)
    K, ridge, back = case["iterations"], 0.005, case["backward"]
    cells = sum(lp.m * lp.n for lp in lps)
    if cells * K * (4 if back else 1) > 6e11:
        return None
    dtype = getattr(torch, case["dtype"])
    if back:
        g = torch.Generator().manual_seed(seed)
        total = sum(lp.n for lp in lps)
        wx = torch.randn(total, generator=g, dtype=dtype).cuda().double()
        wo = torch.rand(len(lps), generator=g, dtype=dtype).cuda().double()
    off = np.concatenate([[0], np.cumsum([lp.n for lp in lps])])
    order = sorted(range(len(lps)), key=lambda b: lps[b].m)
    parts = [None] * len(lps)
    rounded = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dtype).double().cuda()
    at = 0
    while at < len(order):
        group = [b for b in order[at:at + 32]]
        at += len(group)
        M, N = max(lps[b].m for b in group), max(lps[b].n for b in group)
        A = torch.zeros(len(group), M, N, dtype=torch.float64, device="cuda")
        c, cl, cu = (torch.zeros(len(group), N, dtype=torch.float64, device="cuda") for _ in range(3))
        rl, rh = (torch.zeros(len(group), M, dtype=torch.float64, device="cuda") for _ in range(2))
        v0 = torch.zeros(len(group), N, dtype=torch.float64, device="cuda")
        at_nz = []
        for k, b in enumerate(group):
            lp = lps[b]
            rows = torch.from_numpy(np.repeat(np.arange(lp.m), np.diff(lp.ap))).cuda()
            cols = torch.from_numpy(lp.ai.astype(np.int64)).cuda()
            at_nz.append((rows, cols))
            A[k, rows, cols] = rounded(lp.ax)
            for t, v in ((c, lp.c), (cl, lp.cl), (cu, lp.cu)):
                t[k, :lp.n] = rounded(v)
            rl[k, :lp.m], rh[k, :lp.m] = rounded(lp.rmin), rounded(lp.rmax)
            v0[k, :lp.n] = 1.0 / math.sqrt(lp.n)
        mul = lambda X, v: torch.bmm(X, v.unsqueeze(2)).squeeze(2)
        with torch.no_grad():
            v = v0
            for _ in range(100):
                u = mul(A.transpose(1, 2), mul(A, v))
                lam = u.norm(dim=1, keepdim=True)
                v = torch.where(lam > 0, u / lam, u)
            eta = torch.where(lam > 0, 0.9 / lam.sqrt(), torch.ones_like(lam)).to(dtype).double()
        leaf = [A, c, cl, cu, rl, rh]
        if back:
            for t in leaf:
                t.requires_grad_(True)
        with torch.set_grad_enabled(back):
            clamp = lambda t, lo, hi: torch.where(t < lo, lo, torch.where(t > hi, hi, t))
            x = clamp(torch.zeros_like(c), cl, cu)
            y = torch.zeros_like(rl)
            At = A.transpose(1, 2)
            for _ in range(K):
                xn = clamp((x - eta * (c + mul(At, y))) / (1.0 + 2.0 * ridge * eta), cl, cu)
                t = y + eta * mul(A, 2.0 * xn - x)
                y = t - eta * clamp(t / eta, rl, rh)
                x = xn
            obj = (c * x).sum(1) + ridge * (x * x).sum(1)
            if back:
                w = torch.zeros_like(c)
                for k, b in enumerate(group):
                    w[k, :lps[b].n] = wx[off[b]:off[b + 1]]
                loss = (w * x).sum() + (wo[torch.tensor(group).cuda()] * obj).sum()
                gA, gc, gcl, gcu, grl, grh = torch.autograd.grad(loss, leaf)
        for k, b in enumerate(group):
            m, n = lps[b].m, lps[b].n
            parts[b] = {"x": x[k, :n].detach(), "y": y[k, :m].detach(), "obj": obj[k].detach()}
            if back:
                parts[b].update(gc=gc[k, :n], gcl=gcl[k, :n], gcu=gcu[k, :n], grmin=grl[k, :m],
                                grmax=grh[k, :m], gax=gA[k][at_nz[k]])
    return {key: torch.stack([p[key] for p in parts]) if key == "obj"
            else torch.cat([p[key] for p in parts]) for key in parts[0]}
