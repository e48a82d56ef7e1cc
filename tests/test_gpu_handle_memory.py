"""Device memory a handle holds: what its solves so far have needed, not what
other precisions and options would."""
import numpy as np
import pytest
import torch

from igaos_gb300 import generators as G

pytestmark = pytest.mark.gpu


def test_handle_holds_what_its_solves_need(native):
    from igaos_gb300 import capi
    lp = G.random_lp(60000, 150000, 750000, 1)
    m, n, nnz = lp.m, lp.n, lp.nnz
    capi.solve_lp(G.random_lp(30, 60, 90, 0), max_iterations=64, time_limit=1e9)  # the library's own
    free = lambda: torch.cuda.mem_get_info()[0]
    mb = 1 << 20
    # both orientations with their indices in FP64 and FP32 (the FP32 rows padded by
    # an eighth at most besides), the vectors; 6 MB for blocks of 2 MB
    created = nnz * (32 + 9) + n * 138 + m * 106 + 6 * mb
    start = free()
    with capi.Problem(lp) as P:
        torch.cuda.synchronize()
        assert start - free() <= created, ((start - free()) / mb, created / mb)
        P.solve(precision="fp64", max_iterations=64, time_limit=1e9)
        fp64 = created + 8 * (7 * n + 8 * m) + 50 * n + 49 * m + 4 * mb  # iterates, dual repair
        assert start - free() <= fp64, ((start - free()) / mb, fp64 / mb)
        P.solve(precision="fp32-refine", max_iterations=64, time_limit=1e9)
        both = fp64 + 4 * (7 * n + 8 * m) + 60 * (n + m) + 4 * mb
        assert start - free() <= both, ((start - free()) / mb, both / mb)
    assert np.isclose(free(), start, atol=4 * mb)
