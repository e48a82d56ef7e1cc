"""The FP32 step rule sums an LP's rows in FP64, and the sums may not depend on
whether the entries are staged in shared memory, which a batch's other LPs and
single values decide (subnormals are read from global memory)."""
import numpy as np
import pytest
import torch

from igaos_gb300 import generators as G
from igaos_gb300.layer import BatchPattern, pdhg_steps, stack_lps

pytestmark = pytest.mark.gpu


def test_steps_do_not_depend_on_the_batch(native):
    """32 rows whose products with the uniform vector cancel: v0 - v0 and
    x v0 - x v0 in two chains (even and odd entries) leave exactly zero, in one
    chain a rounding error that the power iteration grows into these rows'
    norm. A subnormal value keeps its CTA's share in global memory: alone
    that is the whole LP, beside a large one (which spreads it over CTAs) other
    rows than these. The norm is the last row's 0.5 either way."""
    n, x = 1600, 2.0 ** -10
    k = np.arange(32)  # rows k and k + 16 share four columns
    rows = np.repeat(k, 4)
    cols = (4 * (k % 16)[:, None] + np.arange(4)).reshape(-1)
    vals = np.tile([1.0, x, -1.0, -x], 32)
    rows = np.concatenate([rows, [32, 33]])
    cols = np.concatenate([cols, [70, 71]])
    vals = np.concatenate([vals, [1e-40, 0.5]])
    order = np.lexsort((rows, cols))
    m = 34
    lp = G.from_triplets(m, n, rows[order], cols[order], vals[order], np.zeros(n), np.zeros(n),
                         np.ones(n), np.zeros(m), np.ones(m))
    large = G.bernoulli_lp(np.random.default_rng(3), 1300, 2600, 0.02, 10.0)
    got = []
    for lps, at in (([lp], 0), ([lp, large], 0), ([large, lp], 1)):
        P = BatchPattern.from_lps(lps, "cuda")
        tau, sigma = pdhg_steps(P, stack_lps(lps, torch.float32, "cuda")[5], 2.0)
        got.append((tau[at].item(), sigma[at].item()))
    assert got[0] == got[1] == got[2], got
    assert got[0] == (np.float32(0.9 / 0.5 / 2.0), np.float32(0.9 / 0.5 * 2.0)), got
