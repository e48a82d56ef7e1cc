"""Host threads in the layer with layouts of different shared memory: the
library calls run without the interpreter lock, and none may change what
another's launch is allowed."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from igaos_gb300 import capi
from igaos_gb300 import generators as G
from igaos_gb300.layer import BatchPattern, stack_lps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_small_and_large_layouts_at_once(native, dtype):
    """Thousands of calls of a few microseconds each (zero matrices: the power
    iteration ends at its first product), so that calls meet between each
    other's steps on the host."""
    lib = capi.lib()
    rng = np.random.default_rng(0)
    keep, calls = [], []
    for m, n, d in ((12, 24, 0.2), (450, 900, 0.02), (12, 30, 0.2), (460, 900, 0.02)):
        lp = G.bernoulli_lp(rng, m, n, d, 10.0)
        P = BatchPattern.from_lps([lp], DEV)
        ax = torch.zeros_like(stack_lps([lp], dtype, DEV)[5])
        tau, sigma = torch.zeros(1, dtype=dtype, device=DEV), torch.zeros(1, dtype=dtype, device=DEV)
        L, s = P.layout(dtype, 1, 1, 0.0), torch.cuda.Stream()
        keep.append((P, ax, tau, sigma, L, s))
        calls.append((C.byref(L), C.c_void_p(ax.data_ptr()), 1.0, C.c_void_p(tau.data_ptr()),
                      C.c_void_p(sigma.data_ptr()), C.c_void_p(s.cuda_stream)))
    torch.cuda.synchronize()
    errors = []

    def loop(args):
        for _ in range(5000):
            if lib.igaos_pdhg_unrolled_steps(*args) != capi.OK:
                errors.append(capi.last_error())
                return

    threads = [threading.Thread(target=loop, args=(a,)) for a in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for _, _, tau, sigma, _, _ in keep:
        assert tau.item() == sigma.item() == 1.0
