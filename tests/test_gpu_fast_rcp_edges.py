"""The fast mode's reciprocal and square root where their integer forms change
course: mantissas next to 1 and 2 (the normalising shift), odd and even
exponents, the ends of the range, and what has no normal result.  Errors in
half-ulps of the result, from the exact residuals 1 - d*y and x - y*y (Dekker's
two-product).  Limits: one rounding, the series' remainder (2^-59.7 and 2^-58
of the result, whose half-ulp is 2^-54 at least) and the guard bits' rounding:
1.03 and 1.3."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def call(pkg, name, x):
    xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    yd = torch.empty_like(xd)
    assert getattr(pkg.load_library(), name)(C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr()), x.size) == 0
    return yd.cpu().numpy()


def split(a):
    t = 134217729.0 * a
    h = t - (t - a)
    return h, a - h


def residual(c, a, b):
    """c - a*b for c near a*b, exact but for the last rounding."""
    p = a * b
    (ah, al), (bh, bl) = split(a), split(b)
    e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    return (c - p) - e


def mantissas():
    rng = np.random.default_rng(5)
    near = np.arange(4096)
    return np.concatenate([1 + near * 2.0**-52, 2 - (near + 1) * 2.0**-52, 1 + near / 4096.0,
                           np.sqrt(2.0) + (near - 2048) * 2.0**-52, rng.uniform(1, 2, 1 << 18)])


@pytest.mark.parametrize("expo", [0, 1, -1022, -1021, 511, 1020, 1021])
def test_reciprocal_within_a_rounding(pkg, expo):
    m = mantissas()
    for sign in (1.0, -1.0):
        y = call(pkg, "gpmood_fast_rcp", sign * np.ldexp(m, expo))
        ym = np.ldexp(sign * y, expo)  # the reciprocal of m
        assert np.isfinite(ym).all()
        assert np.abs(residual(1.0, m, ym) / m / (np.spacing(ym) / 2)).max() <= 1.03


def test_reciprocals_that_are_not_normal(pkg):
    tiny, big = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    edge = np.array([2.0**1022, np.nextafter(2.0**1022, np.inf)])  # the seed, within 2^-19.9
    zero = np.array([1.5 * 2.0**1022, 2.0**1023, big])  # subnormal reciprocals
    nan = np.array([0.0, tiny / 2, 5e-324, np.inf, np.nan])
    for s in (1.0, -1.0):
        assert np.abs(call(pkg, "gpmood_fast_rcp", s * edge) - s * tiny).max() <= 2.0**-19.9 * tiny
        y = call(pkg, "gpmood_fast_rcp", s * zero)
        assert (y == 0).all() and (np.signbit(y) == (s < 0)).all(), y
        assert np.isnan(call(pkg, "gpmood_fast_rcp", s * nan)).all()
    assert (call(pkg, "gpmood_fast_rcp", np.array([tiny, -tiny])) == [2.0**1022, -(2.0**1022)]).all()


@pytest.mark.parametrize("expo", [0, 1, -1022, -1021, 510, 511, 1022, 1023])
def test_root_within_a_rounding(pkg, expo):
    m = mantissas()
    y = call(pkg, "gpmood_fast_sqrt", np.ldexp(m, expo))
    odd = expo & 1
    x, ym = m * (1 + odd), np.ldexp(y, -((expo - odd) // 2))  # x in [1, 4), ym its root
    assert np.isfinite(ym).all()
    assert np.abs(residual(x, ym, ym) / (2 * ym) / (np.spacing(ym) / 2)).max() <= 1.3


def test_roots_that_are_not_normal(pkg):
    x = np.array([0.0, -0.0, 5e-324, np.finfo(np.float64).tiny / 2, -1.0, -np.inf, np.inf, np.nan])
    assert np.isnan(call(pkg, "gpmood_fast_sqrt", x)).all()
