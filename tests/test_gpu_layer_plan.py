"""How the layer's launches are laid out (csrc/unrolled.cu, plan()): CTAs per
instance and per SM, the backward's two register budgets, and the backward that
leaves costs and bounds in global memory."""
import ctypes as C
import json
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import ROOT
from igaos_gb300 import capi
from igaos_gb300 import generators as G
from igaos_gb300.layer import BatchPattern, UnrolledPDHG, stack_lps
from oracle import unrolled_dense as U
from test_gpu_unrolled import DEV, RIDGE, relerr, run

pytestmark = pytest.mark.gpu
KEYS = ("ctas", "threads", "per_sm", "smem", "variant", "lean")


def plan(lps, dtype, which):
    P = BatchPattern.from_lps(lps, DEV)
    L, out = P.layout(dtype, 10, 5, 0.005), (C.c_int * len(KEYS))()
    capi._check(capi.lib().igx_unrolled_plan(C.byref(L), which, out))
    return dict(zip(KEYS, out))


def bernoulli(m, density, seed=0):
    return G.bernoulli_lp(np.random.default_rng(seed), m, 2 * m, density, 10.0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_many_small_lps_fill_the_sms(native, dtype, which):
    """An LP of 24 columns takes a few KB and four warps: at 128 registers a
    thread an SM holds four such CTAs, at 64 eight."""
    p = plan([bernoulli(12, 0.2)] * 2000, dtype, which)
    assert p["ctas"] == 1 and p["threads"] == 128
    assert p["per_sm"] >= 8, p
    assert p["smem"] <= 24 * 1024, p


def test_one_cta_per_sm_counts_as_one(native):
    """16 warps at 128 registers fill an SM's registers."""
    p = plan([bernoulli(400, 0.005)] * 100, torch.float32, 2)
    assert p["ctas"] == 1 and p["threads"] == 512 and p["variant"] == 0
    assert p["per_sm"] == 1, p


def test_plans_do_not_depend_on_earlier_calls(native):
    code = """
import json, sys
sys.path[:0] = [%r, %r]
import torch
from test_gpu_layer_plan import bernoulli, plan
lps = {"few warps": [bernoulli(40, 0.6)] * 40, "many": [bernoulli(500, 0.02)] * 40,
       "wide": [bernoulli(1300, 0.01)] * 40}
names = sorted(lps, reverse=len(sys.argv) > 1)
out = {n: [plan(lps[n], d, w) for d in (torch.float32, torch.float64) for w in range(3)] for n in names}
print(json.dumps(out, sort_keys=True))
""" % (ROOT, ROOT + "/tests")
    got = [subprocess.run([sys.executable, "-c", code, *extra], capture_output=True, text=True, check=True)
           .stdout.splitlines()[-1] for extra in ([], ["reversed"])]
    assert json.loads(got[0]) == json.loads(got[1])


def first_results(lps, dtype):
    """Outputs and gradients of the first LP of a batch."""
    P, lp = BatchPattern.from_lps(lps, DEV), lps[0]
    data = [t.requires_grad_(True) for t in stack_lps(lps, dtype, DEV)]
    tau = torch.full((len(lps),), 0.03, dtype=dtype, device=DEV)
    x, y, obj = UnrolledPDHG.apply(*data, tau, tau, P, 30, 8, 0.005)
    grads = torch.autograd.grad((x * x).sum() + y.sum() + obj.sum(), data)
    sizes = (lp.n, lp.n, lp.n, lp.m, lp.m, lp.nnz)
    return [x[:lp.n], y[:lp.m], obj[:1]] + [g[:k] for g, k in zip(grads, sizes)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_register_budgets_agree(native, dtype):
    """The same LP alone and among enough of its size for the other kernel."""
    lp, other = bernoulli(100, 0.05, 1), bernoulli(100, 0.05, 2)
    many = [lp] + [other] * 1500
    assert plan([lp], dtype, 2)["variant"] == 0 and plan(many, dtype, 2)["variant"] == 1
    assert all(torch.equal(a, b) for a, b in zip(first_results([lp], dtype), first_results(many, dtype)))


@pytest.mark.parametrize("dtype,density", [(torch.float64, 0.157), (torch.float32, 0.2955)])
def test_lean_backward(native, dtype, density):
    """LPs just past what one CTA holds with their costs and bounds: bit for bit
    as beside a larger one, whose launch spreads them over a cluster, and in FP64
    against the dense oracle."""
    lp = bernoulli(150, density, 4)
    many, beside = [lp] * 400, [lp] * 3 + [bernoulli(700, 0.03, 5)]
    assert plan(many, dtype, 2)["ctas"] == plan(many, dtype, 2)["lean"] == 1, lp.nnz
    assert plan(beside, dtype, 2)["lean"] == 0
    assert all(torch.equal(a, b) for a, b in zip(first_results(many, dtype), first_results(beside, dtype)))
    if dtype == torch.float64:
        P, fw, g, w, tau, sigma = run(many, 40, 9)
        out, rg = U.gradients(lp, tau[0], sigma[0], 40, RIDGE, gx=w["x"][:lp.n], gy=w["y"][:lp.m],
                              gobj=w["obj"][0])
        assert relerr(fw["x"][:lp.n], out["x"]) <= 1e-10
        for k, n in (("c", lp.n), ("cl", lp.n), ("cu", lp.n), ("rmin", lp.m), ("rmax", lp.m), ("ax", lp.nnz)):
            assert relerr(g[k][:n], rg[k]) <= 1e-8, k
