"""The FP64 dual step divides by sigma with a reciprocal and a remainder step; the
quotient is the correctly rounded one, on operands whose exact quotient lies as
close to the middle of two doubles as quotients can."""
from fractions import Fraction
import random

import numpy as np
import pytest
import torch

from igaos_gb300 import generators as G
from igaos_gb300.layer import BatchPattern, UnrolledPDHG, stack_lps

pytestmark = pytest.mark.gpu
DEV = "cuda"


def hard_quotients(count, seed=0):
    """(z, sigma, quotient) with t = fl(sigma z) and t / sigma = m / 2^54 (1 +- 1 / (sigma
    m)) in integers, m = -+ sigma^-1 mod 2^54 odd and of 54 bits. sigma and the
    quotient just below a power of two, where a product with the rounded reciprocal
    is furthest off, in its last places."""
    rng, out = random.Random(seed), []
    while len(out) < count:
        s = rng.randrange(2 ** 53 - 2 ** 49 + 1, 2 ** 53, 2)
        sign = rng.choice((1, -1))
        m = (-sign * pow(s, -1, 2 ** 54)) % 2 ** 54
        if m < 2 ** 54 - 2 ** 50:
            continue
        t = (s * m + sign) // 2 ** 54
        z = float(Fraction(t, s))
        for k in range(-2, 3):
            v = z + k * float(np.spacing(z))
            if float(s) * v == float(t):  # (one rounding)
                out.append((v, float(s), Fraction(t, s)))
                break
    return out


def test_dual_step_quotients_are_correctly_rounded(native):
    """One iteration from x = 0.5 of a 1 x 1 LP without row bounds: y is the
    remainder t - sigma fl(t / sigma), exact in FP64."""
    cases = hard_quotients(1000)
    one = np.ones(1)
    lps = [G.from_triplets(1, 1, [0], [0], [2.0 * z], 0 * one, 0.5 * one, 0.5 * one, -np.inf * one, np.inf * one)
           for z, _, _ in cases]
    P = BatchPattern.from_lps(lps, DEV)
    sigma = torch.tensor([s for _, s, _ in cases], dtype=torch.float64, device=DEV)
    x, y, obj = UnrolledPDHG.apply(*stack_lps(lps, torch.float64, DEV), torch.ones_like(sigma), sigma, P, 1, 1,
                                   0.0)
    for (z, s, exact), got in zip(cases, y.cpu().numpy()):
        t, q = Fraction(float(s * z)), Fraction(float(exact))
        assert Fraction(float(got)) == t - Fraction(s) * q, (z, s)
