"""The division and square root of the PLAIN march for operands away from the
ends of the range (march_common.cuh: rcp_near, div_near, sqrt_near), restated
with exact fused operations, against IEEE binary32, over the operands the march
meets and for every estimate the hardware may return: rcp.approx is specified
to 1 unit, rsqrt.approx to 2^-22.9, taken here as -2 to +2 units.

One Newton step leaves a relative error of the estimate's squared, (2 * 2^-23)^2
= 2^-44, so its rounding would be wrong where the true value lies within 2^-20 of
a unit from the middle of two floats; the residual of the second step, of the
quotient and of the root is exact and leaves 2^-22 of a unit.  The bar is 5 in 10^6, and none off by more
than the last bit."""
import numpy as np
import pytest

N = 400_000
BAR = 5 * N // 1_000_000


def _fma(a, b, c):
    return (a.astype(np.longdouble) * b.astype(np.longdouble) + c.astype(np.longdouble)).astype(np.float32)


def _off_by(v, units):
    return (v.view(np.int32) + units).view(np.float32)


def _rcp_step(y, r):
    return _fma(r, _fma(-y, r, np.ones_like(y)), r)


def _rcp_once(y, units):
    return _rcp_step(y, _off_by((1.0 / y.astype(np.float64)).astype(np.float32), units))


def _rcp_near(y, units):
    return _rcp_step(y, _rcp_once(y, units))


def _div_near(x, y, units):
    r = _rcp_once(y, units)
    q = x * r
    return _fma(_fma(-q, y, x), r, q)


def _sqrt_near(x, units):
    half = np.float32(0.5)
    inside = x.view(np.uint32) - np.uint32(0x00800000) < np.uint32(0x7F000000)
    s = np.where(inside, x, np.float32(1.0))
    y = _off_by((1.0 / np.sqrt(s.astype(np.float64))).astype(np.float32), units)
    g, h = s * y, half * y
    e = _fma(-g, h, np.full_like(s, half))
    g, h = _fma(g, e, g), _fma(h, e, h)
    g = _fma(_fma(-g, g, s), h, g)
    return np.where(inside, g, x)


def _close(got, want, name):
    off = got != want
    assert off.sum() <= BAR, (name, int(off.sum()))
    assert (np.abs(got - want) <= np.spacing(np.abs(want))).all(), name


DIVISORS = {
    "remap": (1e-5, 1.0, -1.0, 1.0),
    "extinction": (1e-6, 0.2, 0.0, 1e5),
    "altitude": (1.2e7, 1.3e7, -1e11, 1e11),
    "radius": (6.36e6, 6.46e6, -6.46e6, 6.46e6),
    "path": (1.0, 1.2e6, 0.0, 1.2e6),
    "angle": (1.0, 3.2, 0.0, 3.2),
    "steps": (1.0, 257.0, 1.0, 2.4e5),
}
ROOTS = {"length": (4.0e13, 4.2e13), "horizon": (0.0, 1.0), "disc": (0.0, 1e12), "angle": (1e-34, 1e-30)}


@pytest.mark.parametrize("units", (-2, -1, 0, 1, 2))
@pytest.mark.parametrize("name", sorted(DIVISORS))
def test_quotient(name, units):
    lo, hi, x0, x1 = DIVISORS[name]
    rng = np.random.default_rng(sorted(DIVISORS).index(name))
    y = rng.uniform(lo, hi, N).astype(np.float32)
    x = rng.uniform(x0, x1, N).astype(np.float32)
    _close(_rcp_near(y, units), np.float32(1.0) / y, name)
    _close(_div_near(x, y, units), x / y, name)


@pytest.mark.parametrize("units", (-2, -1, 0, 1, 2))
@pytest.mark.parametrize("name", sorted(ROOTS))
def test_root(name, units):
    lo, hi = ROOTS[name]
    x = np.random.default_rng(sorted(ROOTS).index(name)).uniform(lo, hi, N).astype(np.float32)
    _close(_sqrt_near(x, units), np.sqrt(x), name)


def test_root_at_the_ends():
    """0, infinity and NaN stay; a subnormal's root (below 1.1e-19) reads as the
    subnormal itself."""
    x = np.array([0.0, np.inf, np.nan, 1.1754944e-38, 1e-40, 3.4e38], np.float32)
    got, want = _sqrt_near(x, 0), np.sqrt(x)
    assert np.array_equal(got[[0, 1, 2, 3, 5]], want[[0, 1, 2, 3, 5]], equal_nan=True)
    assert abs(got[4] - want[4]) <= 1.1e-19
