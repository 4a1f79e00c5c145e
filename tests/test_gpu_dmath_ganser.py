"""The three functions of the settling chain's Ganser iteration
(f3d_dmath_eval, ops 4 to 6), as the iteration calls them, against extended
precision (numpy longdouble: 64-bit significand on x86, IEEE quad on Arm).

Bounds, from the operations (u = 2^-53):
 * 1/x: the third-order step's error is the cube of the approximation's (about
   2^-20), and the last multiply-add rounds once: 1.02 u.
 * 1/sqrt(x): 2.5 times that cube; the product x*y rounded before the
   residual (its error enters halved, u/2 * 1) and the last rounding: 1.6 u.
 * x^(0.6567-1): the two table values (CUDA's pow and exp2, 2 and 1 ulp, an ulp
   being at most 2 u), their product (u), the last rounding (u) and the series
   (its next term: 0.1 u) with its own roundings, below 2^-8 u:
   8.2 u.
Arguments: the iteration's range, binade edges, the edges of the table's
intervals, and both sides of the ranges beyond which CUDA's own functions are
called (1 ulp for 1/x and sqrt by IEEE, 1 ulp for rsqrt, 2 for pow)."""
import numpy as np
import pytest

import fall3d_gb300 as F

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
A = np.longdouble(0.6567 - 1.0)  # the binary64 value the iteration uses


def _around(v):
    v = np.asarray(v, dtype=np.float64)
    return np.concatenate([v, np.nextafter(v, 0.0), np.nextafter(v, np.inf)])


def _args(kmin, kmax):
    r = np.random.default_rng(9)
    k = np.arange(kmin, kmax + 1)
    mantissas = 1.0 + np.arange(257) / 256.0  # interval edges
    centres = 1.0 + (np.arange(256) + 0.5) / 256.0
    return np.concatenate([10.0 ** r.uniform(-8, 9, 200000), r.uniform(1.0, 4.0, 200000), _around(2.0 ** k),
                           _around(mantissas), _around(centres), _around(mantissas * 2.0 ** kmin),
                           _around(mantissas * 2.0 ** (kmax - 1)), _around([2.0 ** kmin, 2.0 ** kmax, 3305.0])])


def _check(y, exact, bound):
    rel = np.abs(y.astype(np.longdouble) - exact) / exact
    assert float(np.max(rel)) <= bound * U, float(np.max(rel)) / U


def test_reciprocal():
    x = _args(-1000, 1000)
    _check(F.dmath_eval(6, x), 1 / x.astype(np.longdouble), 1.02)


def test_reciprocal_square_root():
    x = _args(-1000, 1000)
    inside = (x >= 2.0 ** -1000) & (x < 2.0 ** 1000)
    y = F.dmath_eval(5, x)
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    _check(y[inside], exact[inside], 1.6)
    _check(y[~inside], exact[~inside], 2.0)


def test_power():
    x = _args(-64, 64)
    y = F.dmath_eval(4, x)
    _check(y, x.astype(np.longdouble) ** A, 8.2)


def test_special_values():
    x = np.array([0.0, np.inf, np.nan, -1.0, 5e-324, 1e308])
    with np.errstate(all="ignore"):
        for op, f in ((6, lambda v: 1.0 / v), (5, lambda v: v ** -0.5), (4, lambda v: v ** float(A))):
            y, t = F.dmath_eval(op, x), f(x)
            assert np.array_equal(np.isnan(y), np.isnan(t)) and np.array_equal(np.isinf(y), np.isinf(t)), op
            ok = np.isfinite(t)
            assert np.all(np.abs(y[ok] - t[ok]) <= 8 * U * np.abs(t[ok])), op
