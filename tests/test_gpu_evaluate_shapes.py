"""igaos_pdhg_evaluate_noalloc over the shapes its row schedule tells apart:
one row, fewer rows than a warp holds, a remainder past a warp and past a
CTA, empty rows and columns, columns of mixed length, rows long enough to
take a whole warp, and points with infinities and NaN. Checked against the
oracle's restatement of the reference evaluate() (src/pdhg/pdhg.cu:173-254).

Tolerances: a sum of k products in any order is within (k + 1) 2^-53 of the
exact one, relative to the sum of the terms' magnitudes (both sides: twice
that, plus a few operations per metric)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("pinf", "dinf", "gap", "op", "od", "prow")


def make_lp(m, n, seed, dense_row=False, dense_col=False, empty=0):
    from igaos_gb300 import generators as G
    rng = np.random.default_rng(seed)
    deg = np.minimum(rng.zipf(1.6, n), m)
    cols = np.repeat(np.arange(n), deg)
    rows = rng.integers(0, m, cols.size)
    if dense_row:
        rows, cols = np.append(rows, np.full(n, m // 2)), np.append(cols, np.arange(n))
    if dense_col:
        rows, cols = np.append(rows, np.arange(m)), np.append(cols, np.full(m, n // 3))
    if empty:
        keep = (rows % 7 != empty % 7) & (cols % 5 != empty % 5)
        rows, cols = rows[keep], cols[keep]
    key = np.unique(cols * m + rows)
    rows, cols = key % m, key // m
    lo = np.where(rng.random(n) < 0.2, -np.inf, rng.uniform(-2.0, 0.0, n))
    hi = np.where(rng.random(n) < 0.2, np.inf, rng.uniform(0.5, 2.0, n))
    b = rng.standard_normal(m)
    rmin = np.where(rng.random(m) < 0.4, -np.inf, b)
    rmax = np.where(rng.random(m) < 0.4, np.inf, b + rng.random(m) * (rng.random(m) < 0.5))
    return G.from_triplets(m, n, rows, cols, rng.standard_normal(rows.size),
                           rng.standard_normal(n), lo, hi, rmin, rmax)


def point(lp, seed, certify):
    rng = np.random.default_rng(seed + 100)
    x = np.clip(rng.standard_normal(lp.n), lp.cl, lp.cu)
    y = rng.standard_normal(lp.m) * (rng.random(lp.m) < 0.7)
    if certify:
        y = np.where((y > 0) & ~np.isfinite(lp.rmax) | (y < 0) & ~np.isfinite(lp.rmin), 0.0, y)
    return x, y


def device_evaluate(native, lp, x, y):
    import torch
    from igaos_gb300 import capi
    d = lambda v, t: torch.from_numpy(np.ascontiguousarray(v, t)).cuda()
    t = [d(getattr(lp, k), np.int32 if k in ("ap", "ai", "cp", "ci") else np.float64)
         for k in ("ap", "ai", "ax", "cp", "ci", "acx", "c", "cl", "cu", "rmin", "rmax")]
    t += [d(x, np.float64), d(y, np.float64), torch.full((6,), -7.0, dtype=torch.float64).cuda()]
    assert native.igaos_pdhg_evaluate_noalloc(
        lp.m, lp.n, *[C.c_void_p(v.data_ptr()) for v in t],
        C.c_void_p(torch.cuda.current_stream().cuda_stream)) == capi.OK
    return dict(zip(KEYS, t[-1].cpu().tolist()))


@pytest.mark.parametrize("m,n,kw", [
    (1, 1, {}), (3, 40, {}), (31, 33, {}), (257, 64, dict(empty=3)),
    (700, 5001, dict(dense_row=True)), (6000, 300, dict(dense_col=True, empty=2)),
    (20001, 30007, dict(dense_row=True, dense_col=True)), (160000, 170001, {})])
def test_shapes(native, orc, m, n, kw):
    import scipy.sparse as sp
    lp = make_lp(m, n, m + n, **kw)
    A = sp.csr_matrix((lp.ax, lp.ai, lp.ap), shape=(m, n))
    absA = abs(A)
    longest = max(np.diff(lp.ap).max(initial=0), np.diff(lp.cp).max(initial=0))
    olp = orc.lp_from(lp)
    for certify in (True, False):
        x, y = point(lp, m, certify)
        want = orc.evaluate(olp, x, y, A @ x, lp.c + A.T @ y)
        got = device_evaluate(native, lp, x, y)
        u = 2.0 ** -52
        fin = lambda v: np.where(np.isfinite(v), np.abs(v), 0.0)
        rt = absA @ np.abs(x) + fin(lp.rmin) + fin(lp.rmax)
        ct = absA.T @ np.abs(y) + np.abs(lp.c)
        e_op = (n + 4) * u * float(np.abs(lp.c) @ np.abs(x))
        e_od = (n + m + longest + 8) * u * float(
            ct @ (fin(lp.cl) + fin(lp.cu)) + np.abs(y) @ (fin(lp.rmin) + fin(lp.rmax)))
        tol = {"pinf": (longest + 8) * u * rt.max(), "prow": (longest + 8) * u * rt.max(),
               "dinf": (longest + 8) * u * ct.max(), "op": e_op, "od": e_od,
               "gap": 2.0 * (e_op + e_od)}
        for k in KEYS:
            if np.isinf(want[k]):
                assert got[k] == want[k], (k, certify)
            else:
                assert abs(got[k] - want[k]) <= tol[k], (k, certify, got[k], want[k], tol[k])


def test_non_finite_points(native, orc):
    """Infinities and NaN in the point: comparisons with a NaN are false, so
    the maxima pass over it, while sums carry it (as FP64 instructions do)."""
    import scipy.sparse as sp
    lp = make_lp(90, 150, 5)
    A = sp.csr_matrix((lp.ax, lp.ai, lp.ap), shape=(90, 150))
    olp = orc.lp_from(lp)
    for at, v in ((7, np.inf), (20, -np.inf), (33, np.nan)):
        x, y = point(lp, 5, True)
        x[at] = v
        with np.errstate(invalid="ignore"):
            want = orc.evaluate(olp, x, y, A @ x, lp.c + A.T @ y)
        got = device_evaluate(native, lp, x, y)
        for k in KEYS:
            same = got[k] == want[k] or (np.isnan(got[k]) and np.isnan(want[k]))
            assert same or abs(got[k] - want[k]) <= 1e-12 * max(1.0, abs(want[k])), (k, v)
