"""The normal distribution function of the network's GELU: the polynomial in
bdda_fno.cu, evaluated here in float32 with fused multiply-adds."""
import math
import os
import re

import numpy as np
import pytest

from conftest import PKG

erfc = np.vectorize(math.erfc)


def _coefficients():
    with open(os.path.join(PKG, "csrc", "bdda_fno.cu")) as f:
        src = f.read()
    body = src[src.index("float2 normal_cdf(float2 z)"):]
    body = body[:body.index("\n}\n")]
    out = [float(v) for v in re.findall(r"both\((-?[0-9.e+-]+)f\)", body)]
    assert len(out) == 12
    return out


def test_fit_of_log2_erfc():
    a = np.linspace(0.0, 6.0, 20001)
    q = np.polyval(_coefficients() + [0.0], a)
    assert np.max(np.abs(np.exp2(q) - erfc(a))) < 5e-9
    assert np.max(np.abs(np.exp2(q) - erfc(a)) / np.maximum(erfc(a), 1e-3)) < 2e-6


@pytest.mark.parametrize("lo,hi", [(-16.0, -8.5), (-8.5, 8.5), (8.5, 16.0)])
def test_float32_evaluation(lo, hi):
    """Within the bound of the rounding: 2^-24 of the last difference, 1 - e, and
    that of e itself (2^-25, its argument's rounding): 1e-7 in all.  From 8.5
    on 0 and 1."""
    f = np.float32
    z = np.linspace(lo, hi, 40001).astype(f)
    a = np.minimum(np.abs(z) * f(0.70710678118654752), f(16))
    fma = lambda x, y, c: (x.astype(np.float64) * y.astype(np.float64) + np.float64(f(c))).astype(f)
    c = _coefficients()
    q = np.full_like(a, f(c[0]))
    for v in c[1:]:
        q = fma(q, a, v)
    e = f(0.5) * np.exp2((q * a).astype(np.float64)).astype(f)
    phi = np.where(z < 0, e, f(1) - e).astype(np.float64)
    true = 0.5 * erfc(-z.astype(np.float64) / math.sqrt(2.0))
    assert np.max(np.abs(phi - true)) < 1e-7
    if abs(lo + hi) > 1:
        assert np.all(phi == (1.0 if lo > 0 else phi)) and np.max(np.where(z < 0, phi, 0)) < 1e-16
