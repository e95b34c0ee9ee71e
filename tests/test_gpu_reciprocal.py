"""The reciprocal of the inverse iteration's pivots against CUDA's division and the
exact quotient: random mantissas over all exponents, powers of two and their
neighbours, both signs, and the values on each side of the window in which it is not the
division itself.

One rounding (0.5 units in the last place) of a value that is off by less than
2^-57 relative, 0.07 units: 0.57; so it differs from the correctly rounded quotient by
one unit at most, and where they differ the quotient lies within 0.07 units of the
middle between two numbers.  Outside the window, and for zeros, infinities and NaN: the same bits."""
from fractions import Fraction

import numpy as np
import pytest

from tests import device_kernels

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_kernels.load("sums", tmp_path_factory.mktemp("recip"))


def _both(lib, x):
    import torch
    X = torch.tensor(x, device="cuda")
    r, q = torch.zeros_like(X), torch.zeros_like(X)
    p = device_kernels.ptr
    assert lib.reciprocals(len(x), p(X), p(r), p(q)) == 0
    return r.cpu().numpy(), q.cpu().numpy()


def _values():
    rng = np.random.default_rng(2)
    e = np.repeat(np.arange(-1022, 1024), 200)
    with np.errstate(over="ignore"):
        x = np.ldexp(1.0 + rng.random(len(e)), e)
    x = np.where(np.isfinite(x), x, 1.0) * rng.choice([-1.0, 1.0], len(x))
    two = np.ldexp(1.0, np.arange(-1022, 1024))
    near = np.concatenate([two, np.nextafter(two, 0), np.nextafter(two, np.inf)])
    # mantissas near 1 and near 2, where the error of an estimate is largest
    m = np.concatenate([1.0 + np.arange(2000) * 2.0 ** -52, 2.0 - np.arange(1, 2000) * 2.0 ** -52,
                        1.0 + np.arange(4096) / 4096.0])
    return np.concatenate([x, near, -near, m, -m * 2.0 ** 300])


def test_within_one_unit_of_the_division(lib):
    x = _values()
    r, q = _both(lib, x)
    np.testing.assert_array_equal(q, 1.0 / x)          # (the division is correctly rounded)
    e = (x.view(np.int64) >> 52) & 0x7ff
    inside = (e >= 23) & (e < 2023)
    np.testing.assert_array_equal(r[~inside], q[~inside])
    ulps = np.abs(r.view(np.int64) - q.view(np.int64))
    assert ulps.max() <= 1
    for k in np.nonzero(ulps)[0][:2000]:
        ulp = Fraction(float(np.spacing(abs(q[k]) * (1 - 2.0 ** -53))))
        assert abs(Fraction(float(r[k])) - 1 / Fraction(float(x[k]))) <= Fraction(57, 100) * ulp
    assert (ulps > 0).mean() <= 0.07 * 2


def test_what_has_no_reciprocal(lib):
    tiny = np.ldexp(1.0, np.array([-1074, -1073, -1030, -1023]))
    x = np.concatenate([tiny, -tiny, [0.0, -0.0, np.inf, -np.inf, np.nan]])
    r, q = _both(lib, x)
    np.testing.assert_array_equal(r, q)
