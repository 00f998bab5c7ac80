"""The reciprocal, quotient and roots of csrc/df64.cuh restated in numpy
(CPU): an FP32 estimate off by up to two units in the last place, refined,
then corrected once by its exactly formed residual.  Checks the series and
its rounding against 64-bit results formed from the pairs' exact sums in
extended steps, not the device code (the GPU parity tests run that).

Tolerance: each correction carries at most four FP32 roundings of a quantity
below 2^-22 of the result, each half a unit (2^-24 relative), and the pair's
low word one rounding of 2^-48: 4 * 2^-46 + 2^-48 < 2^-43.9 in the worst
case; the root mean square is far below, at most 2^-47.5."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

F = np.float32


def fma(a, b, c):
    """FP32 fused multiply-add: the product is exact in FP64."""
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(F)


def pairs(n, seed, lo=-30, hi=30):
    rng = np.random.default_rng(seed)
    v = np.ldexp(1.0 + rng.random(n), rng.integers(lo, hi, n))
    v[:4] = (1.0, 2.0 ** lo, np.nextafter(2.0, 1.0), 2.0 ** hi)
    h = v.astype(F)
    return h, (v - h).astype(F)


def estimate(y, seed):
    rng = np.random.default_rng(seed)
    y = y.astype(F)
    return (y.view(np.int32) + rng.integers(-2, 3, y.size).astype(np.int32)).view(F)


def corrected(y, s, t):
    hi = fma(s, t, y)
    return hi, fma(s, t, y - hi)


def refined_rcp(bh, seed):
    y0 = estimate(1.0 / bh.astype(np.float64), seed)
    return fma(y0, fma(-bh, y0, F(1)), y0)


def refined_rsqrt(ah, seed):
    y0 = estimate(1.0 / np.sqrt(ah.astype(np.float64)), seed)
    return fma(F(0.5) * y0, fma(-ah, y0 * y0, F(1)), y0)


def df_rcp(bh, bl):
    y = refined_rcp(bh, 1)
    e = fma(-bl, y, fma(-bh, y, F(1)))
    return corrected(y, y, fma(e, e, e))


def df_div(ah, al, bh, bl):
    y = refined_rcp(bh, 2)
    e = fma(-bl, y, fma(-bh, y, F(1)))
    q = ah * y
    r = fma(-bh, q, ah) + fma(-bl, q, al)
    return corrected(q, y, fma(r, e, r))


def df_rsqrt(ah, al):
    y = refined_rsqrt(ah, 3)
    s = y * y
    sl = fma(y, y, -s)
    e = fma(-ah, s, F(1)) + fma(-al, s, -ah * sl)
    return corrected(y, F(0.5) * y, fma(F(0.75) * e, e, e))


def df_sqrt(ah, al):
    y = refined_rsqrt(ah, 4)
    x = ah * y
    r = fma(-x, x, ah) + al
    return corrected(x, F(0.5) * y, r)


def residuals(fn):
    """Relative errors, exactly, from rational residuals."""
    n = 4000
    ah, al = pairs(n, 11)
    bh, bl = pairs(n, 12)
    h, l = {"rcp": lambda: df_rcp(bh, bl), "div": lambda: df_div(ah, al, bh, bl),
            "rsqrt": lambda: df_rsqrt(ah, al), "sqrt": lambda: df_sqrt(ah, al)}[fn]()
    out = []
    for i in range(n):
        a, b = Fraction(float(ah[i])) + Fraction(float(al[i])), Fraction(float(bh[i])) + Fraction(float(bl[i]))
        r = Fraction(float(h[i])) + Fraction(float(l[i]))
        # r = exact (1 + d): d from the defining equation, to first order in d
        d = {"rcp": lambda: r * b - 1, "div": lambda: r * b / a - 1,
             "rsqrt": lambda: (r * r * a - 1) / 2, "sqrt": lambda: (r * r / a - 1) / 2}[fn]()
        out.append(float(d))
    return np.abs(np.array(out))


@pytest.mark.parametrize("fn", ["rcp", "div", "rsqrt", "sqrt"])
def test_error_of_the_corrected_estimates(fn):
    e = residuals(fn)
    assert e.max() < 2.0 ** -43.9, np.log2(e.max())
    assert np.sqrt(np.mean(e * e)) < 2.0 ** -47.5, np.log2(np.sqrt(np.mean(e * e)))


def test_special_arguments():
    """1 stays exact, and the limiter's smallest denominator, 1e-36, has a
    finite reciprocal."""
    one, zero = np.ones(1, F), np.zeros(1, F)
    assert df_rcp(one, zero)[0][0] + df_rcp(one, zero)[1][0] == 1
    h = np.array([1e-36], F)
    r = df_rcp(h, (np.array([1e-36]) - h).astype(F))
    assert np.isfinite(r[0][0]) and abs(float(r[0][0]) * 1e-36 - 1) < 1e-6
