"""Batched solve at the edges of its classes (threads of a CTA, what of an
instance is held in shared memory): one row, sizes around 128, 256 and 512,
more rows than columns, empty rows and columns, dense LPs whose matrix fits
without the iterates and LPs that are read from global memory. Every answer
against the single-LP FP64 engine at the same tolerance (2e-5, the bar of the
other batch tests), and the whole batch bit for bit against the same LPs in
another order with others beside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lp_of(m, n, density, seed, gaps=False):
    from igaos_gb300 import generators as G
    rng = np.random.default_rng(seed)
    A = rng.random((m, n)) < density
    A[rng.integers(0, m), :] |= rng.random(n) < 0.3
    if gaps:
        A[::5] = False
        A[:, 2::7] = False
    cols, rows = np.nonzero(A.T)
    vals = rng.standard_normal(rows.size)
    xs = rng.uniform(0.0, 5.0, n)
    b = np.bincount(rows, weights=vals * xs[cols], minlength=m)
    rmin = np.where(np.arange(m) < m // 2, b, -np.inf)
    rmax = np.where(np.arange(m) < m // 2, b, b + rng.random(m))
    return G.from_triplets(m, n, rows, cols, vals, rng.standard_normal(n), np.zeros(n),
                           np.full(n, 5.0), rmin, rmax)


SHAPES = [(1, 1, 1.0), (3, 127, 0.1), (4, 128, 0.1), (5, 129, 0.1), (128, 60, 0.05),
          (129, 33, 0.08), (20, 256, 0.03), (30, 257, 0.03), (40, 511, 0.02), (60, 513, 0.02),
          (530, 90, 0.02), (64, 1100, 0.01)]
DENSE = [(160, 230, 0.35), (90, 300, 0.8), (130, 420, 0.7)]  # matrix alone; global memory


def test_classes_against_single_solves(native):
    from igaos_gb300 import capi
    lps = [lp_of(m, n, d, 7 + k, gaps=k % 3 == 2) for k, (m, n, d) in enumerate(SHAPES + DENSE)]
    out = capi.solve_batch(lps, tolerance=1e-6, max_iterations=200000)
    for lp, r in zip(lps, out):
        want = capi.solve_lp(lp, tolerance=1e-6, time_limit=60.0, precision="fp64")
        assert r["status_name"] == want["status_name"] == "near-optimal", (lp.m, lp.n, r, want["message"])
        assert abs(r["objective"] - want["objective"]) <= 2e-5 * max(1.0, abs(want["objective"])), (lp.m, lp.n)
    more = [lp_of(70, 140, 0.05, 99), lp_of(200, 520, 0.02, 98)]
    back = capi.solve_batch(more + lps[::-1], tolerance=1e-6, max_iterations=200000)[2:][::-1]
    for lp, a, b in zip(lps, out, back):
        if a["finished_fp64"] or b["finished_fp64"]:
            continue
        assert a["iterations"] == b["iterations"], (lp.m, lp.n)
        assert np.array_equal(a["x"], b["x"]) and np.array_equal(a["y"], b["y"]), (lp.m, lp.n)


@pytest.mark.parametrize("m,n", [(40, 29000), (30, 66000)])
def test_instances_wider_than_the_gathered_vectors_shared_memory(native, m, n):
    """Beside an instance of the same class whose gathered vectors fit."""
    from igaos_gb300 import capi
    lps = [lp_of(m, n, 2e-3, 5), lp_of(130, 420, 0.7, 6)]
    out = capi.solve_batch(lps, tolerance=1e-6, max_iterations=200000)
    for lp, r in zip(lps, out):
        want = capi.solve_lp(lp, tolerance=1e-6, time_limit=60.0, precision="fp64")
        assert r["status_name"] == want["status_name"] == "near-optimal", (lp.m, lp.n, r, want["message"])
        assert abs(r["objective"] - want["objective"]) <= 2e-5 * max(1.0, abs(want["objective"])), (lp.m, lp.n)
