"""The series of gpp_far.cu on the CPU: for wtilde anywhere in a box (its
corners among them) and wx at the distance where a pair starts to be far and
beyond, on both sides, the Chebyshev expansion with the kernel's number of
terms equals 1 / (wx - wtilde) to the precision it stands for (2^-53 of the
largest term for FP64, 2^-48 for the mixed path), and every term is within
the bound R^-k that its level of precision rests on."""
import math
import os
import re

import numpy as np
import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "doe-csfg-hackathon_gb300", "csrc")


def _constants():
    text = open(os.path.join(CSRC, "gpp_far.cu")).read()
    fp64_r, high, low = map(float, re.search(
        r"z\.R = !mixed \? ([\d.]+) : [^?]*\? ([\d.]+) : ([\d.]+);", text).groups())
    mixed_b, fp64_b = map(float, re.search(r"z\.bits = mixed \? ([\d.]+) : ([\d.]+);", text).groups())
    return {"fp64": (fp64_r, fp64_b, 53), "mixed": (low, mixed_b, 48), "mixed, high R": (high, mixed_b, 48)}


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed, high R"])
@pytest.mark.parametrize("a,b,v", [(0.5, 2.0, 0.05), (-3.0, 1.0, 0.0), (0.2, 0.3, 0.4), (5.0, 60.0, 1.0)])
def test_series_reaches_the_working_precision(precision, a, b, v):
    R, bits, want = _constants()[precision]
    K = math.ceil(bits / math.log2(R))
    assert K <= 64  # the plan's table of terms
    z0, hw = 0.5 * (a + b), 0.5 * (b - a)
    h = max(hw + v, 1.02 * hw)
    corner = complex(hw / h, v / h)
    s = 0.5 * (abs(corner - 1) + abs(corner + 1))
    rho = s + math.sqrt(max(s * s - 1, 0.0))
    r = R * rho
    d = h * 0.5 * (r + 1 / r)
    rng = np.random.default_rng(3)
    re_ = np.concatenate([rng.uniform(a, b, 400), [a, a, b, b, z0]])
    im_ = np.concatenate([rng.uniform(-v, v, 400), [-v, v, -v, v, v]])
    # In extended precision, so that the error is the series' own.
    ld = np.longdouble
    w = re_.astype(ld) + 1j * im_.astype(ld)
    z = (w - ld(z0)) / ld(h)
    for x in [z0 + d, z0 - d, z0 + 1.3 * d, z0 - 4 * d, z0 + 50 * d]:
        u = (ld(x) - ld(z0)) / ld(h)
        sq = np.copysign(np.sqrt((u - 1) * (u + 1)), u)
        q = 1 / (u + sq)
        total = np.zeros_like(z)
        prev, cur = z, np.ones_like(z)  # T_-1 = T_1, T_0
        for k in range(K):
            term = cur * (1 if k == 0 else 2) * q ** k / (ld(h) * sq)
            assert np.all(np.abs(cur) * abs(q) ** k <= R ** -k * (1 + 1e-9))
            total += term
            prev, cur = cur, 2 * z * cur - prev
        exact = 1 / (ld(x) - w)
        # The terms left out: 2 R^-K R / (R - 1) of the first one's scale, and
        # the rounding of the sum here (K terms of 2^-63 at least).
        scale = 1 / abs(ld(h) * sq)
        assert np.max(np.abs(total - exact)) <= scale * (2.0 ** -want + K * 2.0 ** -60)
