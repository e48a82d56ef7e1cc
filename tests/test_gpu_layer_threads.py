"""Two host threads in the layer with layouts of different shared memory: the
library calls run without the interpreter lock, and neither may change what
the other's launch is allowed. Results against the same calls one after
another, bit for bit."""
import threading

import numpy as np
import pytest
import torch

from igaos_gb300 import generators as G
from igaos_gb300.layer import BatchPattern, UnrolledPDHG, pdhg_steps, stack_lps

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_small_and_large_layouts_at_once(native, dtype):
    def calls(lp):
        """Steps, and a forward and backward of one iteration, of one LP."""
        P = BatchPattern.from_lps([lp], DEV)
        data = [t.requires_grad_(True) for t in stack_lps([lp], dtype, DEV)]

        def go():
            tau, sigma = pdhg_steps(P, data[5])
            x, y, obj = UnrolledPDHG.apply(*data, tau, sigma, P, 1, 1, 0.005)
            return (tau, x, y, *torch.autograd.grad(x.sum() + obj.sum(), data))
        return go

    rng = np.random.default_rng(0)
    # shared memory of about 10 KB, 60 to 120 KB and 100 to 220 KB a pass
    work = [calls(G.bernoulli_lp(rng, m, n, d, 10.0))
            for m, n, d in ((12, 24, 0.2), (250, 500, 0.04), (450, 900, 0.02))]
    want = [w() for w in work]
    torch.cuda.synchronize()
    errors, got = [], [None] * len(work)

    def loop(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(400):
                    got[k] = work[k]()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # (the launch's error, where a size was refused)
            errors.append((k, e))

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for g, w in zip(got, want):
        assert all(torch.equal(a, b) for a, b in zip(g, w))
