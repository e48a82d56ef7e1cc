"""Ruiz factors where the column sweep's quotients leave the reciprocal path
(operands hundreds of binades from 1), with explicit zeros and rows of zeros:
bit-equal to the oracle's loops (src/pdhg/pdhg.cu:474-490)."""
import dataclasses

import numpy as np
import pytest

from igaos_gb300 import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decades", [3, 60, 200, 290])
@pytest.mark.parametrize("shape", [(1, 1, 0), (33, 70, 300), (400, 900, 5000)])
def test_factors_are_the_oracles(native, orc, shape, decades):
    from igaos_gb300 import capi
    lp = G.random_lp(*shape, 5)
    rng = np.random.default_rng(6)
    k = lp.ax.shape[0]
    ax = 10.0 ** rng.uniform(-decades, decades, k) * rng.choice([-1.0, 1.0], k)
    if k > 10:
        ax[rng.random(k) < 0.1] = 0.0
        ax[: lp.ap[1]] = 0.0  # a row of zeros
    cp, ci, acx = orc.transpose(lp.m, lp.n, lp.ap, lp.ai, ax)
    lp = dataclasses.replace(lp, ax=ax, cp=cp, ci=ci, acx=acx)
    rdr, rdc = orc.ruiz(orc.lp_from(lp))
    with capi.Problem(lp) as P:
        dr, dc = P.scaling()
    assert np.array_equal(dr, rdr)
    assert np.array_equal(dc, rdc)
