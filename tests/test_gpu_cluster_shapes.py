"""Cluster sizes and storage of the small-LP attempt kernel (csrc/cluster.cuh).

FP64 sums are those of the grid-wide kernels whatever the cluster's size: the
state after a run of iterations is equal bit for bit with IGAOS_PDHG_CLUSTER=0.
FP32 attempts are held to the oracle's iteration (src/pdhg/pdhg.cu:748-799), also
where the iterates stay in global memory (the last shape, whose replicas leave
no room for them).
"""
import numpy as np
import pytest

from igaos_gb300 import generators as G

pytestmark = pytest.mark.gpu

# (m, n, entries): one item per orientation; one CTA; more virtual warps than one
# CTA's; several items per virtual warp; FP64 partials of more than 32 groups; the
# largest
SHAPES = [(1, 1, 1), (20, 31, 60), (33, 65, 400), (300, 700, 2500), (1100, 2100, 30000),
          (2000, 5000, 20000), (300, 10000, 12000), (6000, 22000, 22000)]


def state(capi, lp, iters, precision):
    with capi.Problem(lp) as P:
        _, eta0, omega0 = P.step_init()
        z = lambda k: np.zeros(k)
        st = dict(x=z(lp.n), y=z(lp.m), xavg=z(lp.n), yavg=z(lp.m), axcur=z(lp.m), eta=eta0,
                  omega=omega0, k=1, hn=0)
        return st, P.iterate(st, iters, precision)


@pytest.mark.parametrize("shape", SHAPES)
def test_fp64_is_the_grid_kernels_bit_for_bit(native, monkeypatch, shape):
    from igaos_gb300 import capi
    m, n, nnz = shape
    lp = G.random_lp(m, n, max(0, nnz - n), 3)
    monkeypatch.setenv("IGAOS_PDHG_CLUSTER", "0")
    _, want = state(capi, lp, 70, "fp64")
    monkeypatch.delenv("IGAOS_PDHG_CLUSTER")
    _, got = state(capi, lp, 70, "fp64")
    for key in ("x", "y", "xavg", "yavg", "axcur"):
        assert np.array_equal(got[key], want[key]), key
    for key in ("eta", "omega", "k", "hn", "attempts"):
        assert got[key] == want[key], key


@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_tracks_the_oracle(native, orc, shape):
    """Five iterations: FP32 rounding (2^-24 per operation, iterates of unit
    scale) stays within the 2e-4 of the other FP32 iteration tests."""
    from igaos_gb300 import capi
    m, n, nnz = shape
    lp = G.random_lp(m, n, max(0, nnz - n), 3)
    olp = orc.lp_from(lp)
    sd = orc.scale(olp, *orc.ruiz(olp))
    st0, got = state(capi, lp, 5, "fp32")
    want, _ = orc.iterate(olp, sd, st0, 5)
    assert got["k"] == want["k"]
    for key in ("x", "y"):
        scale = max(1.0, float(np.max(np.abs(want[key]))))
        assert np.max(np.abs(got[key] - want[key])) <= 2e-4 * scale, key
