"""The FP64 Ewald path's erfcx (csrc/ewald.cu, erfcx_poly): the coefficients read from
the kernel source, evaluated in 60-digit arithmetic, give erfcx to the stated
remainder, and in FP64 to a few roundings (host only; the tensors' own tests bound
the device path at 1e-10)."""
import os
import re
from decimal import Decimal, getcontext

import numpy as np

from conftest import ROOT

getcontext().prec = 60
PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494")


def _table():
    with open(os.path.join(ROOT, "pybrown_b200", "csrc", "ewald.cu")) as f:
        src = f.read()
    body = src[src.index("__constant__ double c_erfcx["):]
    body = body[:body.index("};")]
    coefs = re.findall(r"-?\d\.\d+e[+-]\d+", body)
    assert len(coefs) == 23 and "c_erfcx[23]" in body
    # the map t = (x - K) / (x + K) of the evaluation
    poly = src[src.index("double erfcx_poly(double x)"):]
    poly = poly[:poly.index("\n}\n")]
    assert "x + 3.5" in poly and "(x - 3.5) * r" in poly and "i < 23" in poly
    return coefs


def _erfcx(x):
    """e^{x^2} erfc(x): the power series of erf below 3, the continued fraction above."""
    x = Decimal(x)
    if x < 3:
        term, total, n = x, x, 0
        while abs(term) > Decimal("1e-58"):
            n += 1
            term *= -x * x / n
            total += term / (2 * n + 1)
        return (x * x).exp() * (1 - 2 * total / PI.sqrt())
    f = x
    for k in range(600, 0, -1):
        f = x + Decimal(k) / 2 / f
    return 1 / (f * PI.sqrt())


def _points():
    return [float(v) for v in np.concatenate([np.linspace(0.0, 8.0, 161), np.geomspace(8.0, 60.0, 40)])]


def test_remainder_of_the_polynomial():
    coefs = [Decimal(float(c)) for c in _table()]  # the doubles that the kernel holds
    for x in _points():
        t = (Decimal(x) - Decimal("3.5")) / (Decimal(x) + Decimal("3.5"))
        p = coefs[0]
        for c in coefs[1:]:
            p = p * t + c
        exact = _erfcx(x)
        # below 6e-17 of the value of (x + K) erfcx, between 0.56 and 3.5, and the
        # coefficients' own roundings: 2^-54 of each, 3.7 in all, of values from 0.56
        assert abs(p / (Decimal(x) + Decimal("3.5")) / exact - 1) < Decimal("4.3e-16"), x


def test_fp64_evaluation():
    coefs = [float(c) for c in _table()]
    for x in _points():
        r = 1.0 / (x + 3.5)
        t = (x - 3.5) * r
        p = coefs[0]
        for c in coefs[1:]:
            p = p * t + c
        # about one rounding of each partial sum (below 1.6 in magnitude past the last
        # few terms) and of r: a dozen of 1.1e-16
        assert abs(Decimal(p * r) / _erfcx(x) - 1) < Decimal("1.4e-15"), x
