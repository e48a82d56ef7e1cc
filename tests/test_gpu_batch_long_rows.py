"""Batched solve of LPs with full rows and columns, and rows of Zipf lengths,
whose slices are staged in steps of decreasing width: in every mode an
instance is held in, against the single-LP FP64 engine (2e-5, the bar of the
other batch tests), and bit for bit in another batch."""
import numpy as np
import pytest

from igaos_gb300 import generators as G
from test_batch_plan_cpu import ALL, MATRIX, OUT, WIDE, pattern, plan

pytestmark = pytest.mark.gpu


def feasible(A, seed):
    rng = np.random.default_rng(seed)
    m, n = A.shape
    cols, rows = np.nonzero(A.T)
    vals = rng.standard_normal(rows.size) / np.sqrt(A.sum(1))[rows]
    xs = rng.uniform(0.0, 5.0, n)
    b = np.bincount(rows, weights=vals * xs[cols], minlength=m)
    eq = np.arange(m) < m // 2
    return G.from_triplets(m, n, rows, cols, vals, rng.standard_normal(n), np.zeros(n), np.full(n, 5.0),
                           np.where(eq, b, -np.inf), np.where(eq, b, b + rng.random(m)))


def zipf_rows(m, n, seed):
    A = pattern(m, n, 0.0, seed=seed)
    rng = np.random.default_rng(seed)
    for i in range(m):
        A[i, rng.choice(n, max(1, n // (1 + i)), replace=False)] = True
    return A


CASES = [(ALL, pattern(40, 100, 0.05, 1)), (ALL, pattern(33, 65, 0.1, 1, 1)), (ALL, pattern(1, 70, 0.1)),
         (ALL, pattern(70, 1, 1.0)), (ALL, pattern(30, 600, 0.02, 2, 2)), (ALL, zipf_rows(64, 200, 2)),
         (ALL, pattern(500, 1250, 0.01, 1)), (MATRIX, pattern(60, 4000, 0.005, 1)),
         (OUT, pattern(200, 5000, 0.005, 4, 3)), (WIDE, pattern(20, 29000, 0.002, 1))]


def test_long_rows_in_every_mode(native):
    from igaos_gb300 import capi
    lps = [feasible(A, 3 + k) for k, (_, A) in enumerate(CASES)]
    assert [int(v) for v in plan(lps)[1]] == [mode for mode, _ in CASES]
    out = capi.solve_batch(lps, tolerance=1e-6, max_iterations=200000)
    for lp, r in zip(lps, out):
        want = capi.solve_lp(lp, tolerance=1e-6, time_limit=60.0, precision="fp64")
        assert r["status_name"] == want["status_name"] == "near-optimal", (lp.m, lp.n, r, want["message"])
        assert abs(r["objective"] - want["objective"]) <= 2e-5 * max(1.0, abs(want["objective"])), (lp.m, lp.n)
    back = capi.solve_batch([feasible(pattern(50, 90, 0.1), 1)] + lps[::-1], tolerance=1e-6,
                            max_iterations=200000)[1:][::-1]
    for lp, a, b in zip(lps, out, back):
        if a["finished_fp64"] or b["finished_fp64"]:
            continue
        assert a["iterations"] == b["iterations"], (lp.m, lp.n)
        assert np.array_equal(a["x"], b["x"]) and np.array_equal(a["y"], b["y"]), (lp.m, lp.n)

