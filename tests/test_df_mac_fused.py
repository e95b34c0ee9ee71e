"""The double-float multiply-add that takes the product's rounding error along
with the TwoSum correction in one FMA, emulated in IEEE float32 on the host.

df_mac(acc, a, b): p = fl(a.hi b.hi), s = fl(acc.hi + p), bb = fl(s - acc.hi),
e = fma(a.hi, b.hi, -bb), e = fma(a.hi, b.lo, e), e = fma(a.lo, b.hi, e),
acc = (s, acc.lo + ((acc.hi - (s - bb)) + e)).

Bound of a K-term sum: every correction is at most 2^-23 S (S = sum |x y|) and
the low word at most K 2^-23 S, so a step rounds by at most (K + 5) 2^-47 S:
K (K + 5) 2^-47 S in all."""
from fractions import Fraction

import numpy as np
import pytest

f32 = np.float32


def _fma(a, b, c):
    """Correctly rounded: TwoSum in float64 of the exact product and the addend, rounded to odd."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    s = p + c
    bb = s - p
    e = (p - (s - bb)) + (c - bb)
    i = s.view(np.int64).copy()
    i = np.where((e != 0) & ((i & 1) == 0), np.where((e > 0) == (s > 0), i + 1, i - 1), i)
    return i.view(np.float64).astype(f32)


def _df_mac(hi, lo, ah, al, bh, bl):
    s = (hi + (ah * bh).astype(f32)).astype(f32)
    bb = (s - hi).astype(f32)
    e = _fma(ah, bh, -bb)
    e = _fma(ah, bl, e)
    e = _fma(al, bh, e)
    e = ((hi - (s - bb).astype(f32)).astype(f32) + e).astype(f32)
    return s, (lo + e).astype(f32)


@pytest.mark.parametrize("terms", [1, 2, 16, 64])
@pytest.mark.parametrize("spread", [0, 6, 12])
def test_sums_stay_at_the_double_float_level(terms, spread):
    rng = np.random.default_rng(terms + spread)
    n = 300
    x, y = (rng.standard_normal((n, terms)) * 10.0 ** rng.uniform(-spread, 0, (n, terms)) for _ in range(2))
    if terms > 1:  # a pair that cancels to a few units in the last place
        x[::3, -1], y[::3, -1] = -x[::3, 0] * (1 + rng.integers(-3, 4, x[::3, 0].size) * 2.0 ** -23), y[::3, 0]
    (xh, xl), (yh, yl) = ((v.astype(f32), (v - v.astype(f32)).astype(f32)) for v in (x, y))
    hi = lo = np.zeros(n, f32)
    for k in range(terms):
        hi, lo = _df_mac(hi, lo, xh[:, k], xl[:, k], yh[:, k], yl[:, k])
    F = lambda v: Fraction(float(v))  # noqa: E731
    for i in range(n):
        prod = [(F(xh[i, k]) + F(xl[i, k])) * (F(yh[i, k]) + F(yl[i, k])) for k in range(terms)]
        err = abs(F(hi[i]) + F(lo[i]) - sum(prod))
        assert err <= terms * (terms + 5) * Fraction(1, 2 ** 47) * sum(abs(v) for v in prod)
