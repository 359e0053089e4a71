"""The multiply-add division of the PLAIN march (march_common.cuh:div_by),
restated with exact fused operations, against IEEE binary32 division, for the
divisors the march knows in advance: the noise, detail and weather scales, the
layer thickness, the sun's cosine, the coverage remap and the constant edges of
the profiles, over the operands they meet.  The estimate is within 1.5 units,
and its residual is exact, so the corrected quotient is off only where the
true one lies within 2^-23 of a unit from the middle of two floats: the bar is
one quotient in 10^6, and none off by more than the last bit."""
import numpy as np
import pytest

N = 400_000


def _fma(a, b, c):
    """fma in binary32: 64-bit mantissas hold the product (48 bits) exactly and
    the sum to 2^-63, far below what a second rounding could notice here."""
    return (a.astype(np.longdouble) * b.astype(np.longdouble) + c.astype(np.longdouble)).astype(np.float32)


def _div_by(x, d, r):
    q = (x * r).astype(np.float32)
    return _fma(_fma(-q, d, x), r, q)


CASES = {
    "base_scale": (4500.0, 4500.0, -4e5, 4e5),
    "detail_scale": (800.0, 800.0, -4e5, 4e5),
    "weather_scale": (32000.0, 32000.0, -4e5, 4e5),
    "any_scale": (1.0, 50000.0, -4e5, 4e5),
    "thickness": (1.0, 12000.0, 0.0, 12000.0),
    "cos_sun": (0.05, 1.0, 0.0, 12000.0),
    "coverage": (0.01, 1.0, -1.0, 1.0),
    "profile": (0.05, 0.8, 0.0, 1.0),
    "radius": (6.36e6, 6.46e6, -6.46e6, 6.46e6),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_multiply_add_division_is_the_ieee_quotient(name):
    lo, hi, x0, x1 = CASES[name]
    rng = np.random.default_rng(sorted(CASES).index(name))
    d = rng.uniform(lo, hi, N).astype(np.float32) if hi > lo else np.full(N, lo, np.float32)
    x = rng.uniform(x0, x1, N).astype(np.float32)
    r = (np.float32(1.0) / d).astype(np.float32)
    want = (x / d).astype(np.float32)
    got = _div_by(x, d, r)
    off = got != want
    assert off.sum() <= max(1, N // 1_000_000), (name, int(off.sum()))
    assert (np.abs(got - want) <= np.spacing(np.abs(want))).all()


def test_constant_edges_of_the_profiles():
    """Every binary32 height on a fine grid through the profiles' own edges."""
    h = np.linspace(0.0, 1.0, N, dtype=np.float32)
    for e0, e1 in ((0.0, 0.07), (1.0, 0.2), (0.0, 0.10), (0.6, 1.0), (0.0, 0.15), (1.0, 0.4), (0.0, 0.20), (1.0, 0.3),
                   (0.0, 0.30), (0.7, 1.0), (0.0, 0.40), (0.0, 0.50), (0.8, 1.0), (0.0, 0.05), (0.95, 0.5), (0.7, 0.9),
                   (0.65, 0.8)):
        a, b = np.float32(e0), np.float32(e1)
        d = np.full(N, b - a, np.float32)
        r = (np.float32(1.0) / d).astype(np.float32)
        x = (h - a).astype(np.float32)
        assert np.array_equal(_div_by(x, d, r), (x / d).astype(np.float32)), (e0, e1)
