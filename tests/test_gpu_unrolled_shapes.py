"""The layer's staging and cluster paths at the sizes where they can go wrong:
slices of 32 rows and their remainders, empty and full rows, rows of more
entries than the counting sort has classes, one LP spread over several CTAs,
LPs whose entries do not fit on chip beside ones whose do. FP64 results
against the dense checker; the sums are the same chains in the same order as
a plain CSR walk, so K iterations stay within the tolerances the other layer
tests use (forward 1e-10, gradients 1e-8)."""
import numpy as np
import pytest
import torch

from igaos_gb300 import generators as G
from igaos_gb300.layer import BatchPattern, UnrolledPDHG, pdhg_steps, stack_lps
from test_gpu_unrolled import DEV, RIDGE, check_against_dense, run

pytestmark = pytest.mark.gpu


def lp_of(m, n, density, seed, dense_row=False, dense_col=False, skip=False):
    rng = np.random.default_rng(seed)
    A = rng.random((m, n)) < density
    if dense_row:
        A[m // 2] = True
    if dense_col:
        A[:, n // 2] = True
    if skip:  # empty rows and columns
        A[::3] = False
        A[:, 1::4] = False
    cols, rows = np.nonzero(A.T)
    vals = rng.standard_normal(rows.size)
    xs = rng.uniform(-1.0, 2.0, n)
    ax = np.bincount(rows, weights=vals * xs[cols], minlength=m)
    lo = np.where(rng.random(n) < 0.3, -np.inf, xs - rng.random(n))
    hi = np.where(rng.random(n) < 0.3, np.inf, xs + rng.random(n))
    rmin = np.where(rng.random(m) < 0.4, -np.inf, ax)
    rmax = np.where(rng.random(m) < 0.3, np.inf, ax + rng.random(m))
    return G.from_triplets(m, n, rows, cols, vals, rng.standard_normal(n), lo, hi, rmin, rmax)


@pytest.mark.parametrize("sizes", [
    [(1, 1, 1.0), (31, 33, 0.2), (32, 64, 0.2), (33, 32, 0.2), (2, 129, 0.5)],
    [(160, 1200, 0.02)],
    [(900, 700, 0.01), (20, 30, 0.3)]])
def test_slices(native, sizes):
    lps = [lp_of(m, n, d, 10 * k, dense_row=k % 2 == 0, dense_col=k % 2 == 1, skip=k == 1)
           for k, (m, n, d) in enumerate(sizes)]
    check_against_dense(lps, K=60, ck=17, tol_fw=1e-10, tol_g=1e-8)


def test_long_rows_in_several_classes(native):
    """Rows past the counting sort's last class keep the slice order."""
    rng = np.random.default_rng(4)
    m, n = 70, 1500
    A = rng.random((m, n)) < rng.uniform(0.6, 1.0, (m, 1))
    cols, rows = np.nonzero(A.T)
    vals = rng.standard_normal(rows.size)
    lp = G.from_triplets(m, n, rows, cols, vals, rng.standard_normal(n), np.zeros(n), np.ones(n),
                         np.full(m, -1.0), np.full(m, 1.0))
    assert np.diff(lp.ap).min() < 1024 < np.diff(lp.ap).max()
    check_against_dense([lp], K=40, ck=16, tol_fw=1e-10, tol_g=1e-8)


def test_beyond_one_cta_and_beyond_the_chip(native):
    """An LP that several CTAs share and one that is read from global memory,
    each alone and in one batch with a small LP: the same results bit for
    bit, and the dense checker's."""
    small, shared, large = lp_of(40, 60, 0.1, 1), lp_of(700, 900, 0.06, 2), lp_of(900, 1100, 0.3, 3)
    check_against_dense([small, shared, large], K=20, ck=8, tol_fw=1e-10, tol_g=1e-8)
    for dtype in (torch.float64, torch.float32):
        tau = torch.full((3,), 0.02, dtype=dtype, device=DEV)
        whole = run([small, shared, large], 20, 8, dtype, tau=tau, sigma=tau)
        for k, lp in enumerate((small, shared, large)):
            P = BatchPattern.from_lps([lp], DEV)
            x, y, obj = UnrolledPDHG.apply(*stack_lps([lp], dtype, DEV), tau[:1], tau[:1], P, 20, 8,
                                           RIDGE)
            at = slice(whole[0].col_off[k], whole[0].col_off[k + 1])
            assert np.array_equal(x.double().cpu().numpy(), whole[1]["x"][at])
            assert obj.double().item() == whole[1]["obj"][k]


def test_steps_of_odd_matrices(native):
    """A zero matrix takes eta = 1; scales far from 1 keep the quotient of
    the norms (one diagonal block: the largest entry is the norm)."""
    for dtype, scales in ((torch.float64, (0.0, 1e-60, 1.0, 1e60)), (torch.float32, (0.0, 1e-12, 1e12))):
        for s in scales:
            n = 40
            lp = G.from_triplets(n, n, np.arange(n), np.arange(n), s * np.linspace(0.5, 1.0, n) ** 4,
                                 np.zeros(n), np.zeros(n), np.ones(n), np.zeros(n), np.ones(n))
            P = BatchPattern.from_lps([lp], DEV)
            tau, sigma = pdhg_steps(P, stack_lps([lp], dtype, DEV)[5], 2.0)
            v = np.full(n, 1.0 / np.sqrt(n))
            d = np.asarray(stack_lps([lp], dtype, "cpu")[5].double())
            lam = 0.0
            for _ in range(100):
                u = d * (d * v)
                lam = np.linalg.norm(u)
                if not lam > 0:
                    break
                v = u / lam
            eta = 0.9 / np.sqrt(lam) if lam > 0 else 1.0
            eps = 1e-13 if dtype == torch.float64 else 2e-7
            assert abs(float(tau[0]) - eta / 2.0) <= eps * eta
            assert abs(float(sigma[0]) - eta * 2.0) <= eps * eta * 2.0
