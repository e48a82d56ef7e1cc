"""Staging plan of the batched solve (csrc/batch.cu): slices of 32 like rows are
padded to their longest; slices that this would more than double are laid in
steps of decreasing width. Host code, no GPU."""
import ctypes as C

import numpy as np
import pytest

from igaos_gb300 import generators as G

WIDE, OUT, MATRIX, ALL = range(4)
CTAS = (6, 4, 2, 1, 1)  # of the classes, per SM


def plan(lps):
    from igaos_gb300 import capi
    k = len(lps)
    arr = lambda v, t: np.ascontiguousarray(v, t)
    m, n = arr([lp.m for lp in lps], np.int32), arr([lp.n for lp in lps], np.int32)
    ap = arr(np.concatenate([lp.ap for lp in lps]), np.int32)
    ai = arr(np.concatenate([lp.ai for lp in lps]), np.int32)
    cls, mode, entries = np.zeros(k, np.int32), np.zeros(k, np.int32), np.zeros(k, np.int64)
    p = lambda a: C.c_void_p(a.ctypes.data)
    capi.lib().igx_batch_plan(k, p(m), p(n), p(ap), p(ai), p(cls), p(mode), p(entries))
    return cls % len(CTAS), mode, entries  # (LPs with long rows have the classes again)


def lp_of(A):
    cols, rows = np.nonzero(A.T)
    m, n = A.shape
    return G.from_triplets(m, n, rows, cols, np.ones(rows.size), np.zeros(n), np.zeros(n), np.ones(n),
                           np.zeros(m), np.ones(m))


def pattern(m, n, density, full_rows=0, full_cols=0, seed=0):
    rng = np.random.default_rng(seed)
    A = rng.random((m, n)) < density
    A[rng.integers(0, m, n), np.arange(n)] = True
    A[m // 3:m // 3 + full_rows] = True
    A[:, n // 3:n // 3 + full_cols] = True
    return A


# (m, n, density), and how the LP is held with one full row
@pytest.mark.parametrize("m,n,density,held", [(40, 100, 0.05, ALL), (120, 300, 0.02, ALL),
                                              (500, 1250, 0.01, ALL), (30, 600, 0.02, ALL),
                                              (60, 4000, 0.005, MATRIX)])
def test_one_full_row_keeps_its_residency(native, m, n, density, held):
    sparse, dense = lp_of(pattern(m, n, density)), lp_of(pattern(m, n, density, full_rows=1))
    cls, mode, entries = plan([sparse, dense])
    assert mode[0] == mode[1] == held, mode
    assert CTAS[cls[1]] > 1 or CTAS[cls[0]] == 1, cls


@pytest.mark.parametrize("seed", range(6))
def test_padding_is_bounded_where_it_costs(native, seed):
    """LPs that are not held whole: at most four times a slice's entries and 160
    (steps hold at most twice a slice's entries behind a unit of 32, and pads are
    kept below twice that), whatever their rows."""
    rng = np.random.default_rng(seed)
    lps = []
    for _ in range(40):
        m, n = (int(np.exp(rng.uniform(np.log(lo), np.log(hi)))) for lo, hi in ((60, 500), (400, 4000)))
        A = pattern(m, n, rng.uniform(0, 0.1), rng.integers(0, 4), rng.integers(0, 4), int(rng.integers(1 << 30)))
        if rng.random() < 0.5:  # rows of Zipf lengths
            A &= rng.random((m, n)) < (1.0 / (1 + rng.permutation(m)))[:, None]
        if rng.random() < 0.3:
            A[rng.random(m) < 0.4] = False
        lps.append(lp_of(A))
    cls, mode, entries = plan(lps)
    assert (mode < ALL).any() and (mode == ALL).any()
    for lp, e, how in zip(lps, entries, mode):
        slices = (lp.m + 31) // 32 + (lp.n + 31) // 32
        if how < ALL:
            assert e <= 4 * 2 * lp.nnz + 160 * slices, (lp.m, lp.n, lp.nnz, e)


def test_like_rows_stay_padded(native):
    """Every row of the same length: the entries themselves, in units of 32."""
    A = np.zeros((64, 160), bool)
    for i in range(64):
        A[i, (np.arange(10) * 16 + i) % 160] = True
    cls, mode, entries = plan([lp_of(A)])
    assert np.all(A.sum(0) == 4)
    assert entries[0] == 2 * A.sum()
