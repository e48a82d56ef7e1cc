"""Which attempt kernel an LP takes: the tests that compare the cluster kernel with
the grid-wide ones say nothing where both runs take the same. A solve on the cluster
launches once per chunk instead of twice per attempt."""
import numpy as np
import pytest

from igaos_gb300 import generators as G
from test_gpu_cluster_shapes import SHAPES, state

pytestmark = pytest.mark.gpu

LARGEST, BEYOND = (300, 14000, 16000), (300, 15000, 17000)  # in FP64
LARGEST32, BEYOND32 = (6000, 20000, 20000), SHAPES[-1]


def launches(capi, monkeypatch, shape, precision, path):
    monkeypatch.setenv("IGAOS_PDHG_CLUSTER", path)
    m, n, nnz = shape
    r = capi.solve_lp(G.random_lp(m, n, max(0, nnz - n), 3), precision=precision, tolerance=1e-13,
                      max_iterations=512, time_limit=1e9)
    return r["launches"], r["iterations"]


@pytest.mark.parametrize("shape", SHAPES + [LARGEST, BEYOND, LARGEST32])
@pytest.mark.parametrize("precision", ["fp64", "fp32-refine"])
def test_path_taken(native, monkeypatch, shape, precision):
    from igaos_gb300 import capi
    auto, its = launches(capi, monkeypatch, shape, precision, "1")
    grid, grid_its = launches(capi, monkeypatch, shape, precision, "0")
    if shape == BEYOND32 or precision == "fp64" and shape in (BEYOND, LARGEST32):
        assert auto == grid, (auto, grid)
    else:
        assert auto / its * 3 < grid / grid_its, (auto, grid, its, grid_its)


def test_largest_fp64_cluster_is_the_grid_kernels_bit_for_bit(native, monkeypatch):
    from igaos_gb300 import capi
    m, n, nnz = LARGEST
    lp = G.random_lp(m, n, nnz - n, 3)
    monkeypatch.setenv("IGAOS_PDHG_CLUSTER", "0")
    _, want = state(capi, lp, 70, "fp64")
    monkeypatch.delenv("IGAOS_PDHG_CLUSTER")
    _, got = state(capi, lp, 70, "fp64")
    for key in ("x", "y", "xavg", "yavg", "axcur"):
        assert np.array_equal(got[key], want[key]), key
    assert all(got[key] == want[key] for key in ("eta", "omega", "k", "hn", "attempts"))
