"""The digits of the long-K tensor-core products and the sums of their groups, as
the device computes them.

Seven digits on the grid 2^-56 of the row's exponent (largest magnitude below
2^E) leave a residual of at most half a grid step, 2^-57; |m_0| <= 256 and
|m_s| <= 128 are exact in half precision, and the sums of 64 products per pair stay
below 2^24.  A row with an infinity or NaN gets an exponent whose products are not finite.

The folds add 7 integers a_u 2^-8u: groups 4-6 (below 2^24 2^-32 = 2^-8) round twice in
float, by at most 2^-32 each; each of the other additions loses nothing but the
rounding of the low word, which stays below 1 (rounding errors of sums below 2^23)
and so rounds by at most 2^-24 each of four times."""
from fractions import Fraction

import numpy as np
import pytest

from tests import device_kernels

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_kernels.load("digits", tmp_path_factory.mktemp("digits"))


def _digits(lib, hi, lo, neg):
    import torch
    dev = torch.device("cuda")
    h, l = torch.tensor(hi, device=dev), torch.tensor(lo, device=dev)
    E = torch.zeros(len(hi), dtype=torch.int32, device=dev)
    d = torch.zeros(len(hi), 7, 64, device=dev)
    p = device_kernels.ptr
    assert lib.digits(len(hi), p(h), p(l), int(neg), p(E), p(d)) == 0
    return E.cpu().numpy().astype(np.int64), d.cpu().numpy().astype(np.float64)


def _rows(rng, rows, exponents):
    x = rng.standard_normal((rows, 64)) * 10.0 ** rng.uniform(-9, 0, (rows, 64))
    x[rng.random((rows, 64)) < 0.1] = 0.0
    x *= 2.0 ** rng.integers(*exponents, (rows, 1))
    hi = x.astype(f32)
    return hi, (x - hi.astype(np.float64)).astype(f32)


@pytest.mark.parametrize("neg", [False, True])
@pytest.mark.parametrize("kind", ["ordinary", "tiny", "subnormal", "huge", "edges"])
def test_digits_reconstruct_to_half_a_grid_step(lib, kind, neg):
    rng = np.random.default_rng(3)
    hi, lo = _rows(rng, 64, {"ordinary": (-20, 20), "tiny": (-124, -100), "subnormal": (-146, -126),
                             "huge": (90, 120), "edges": (0, 1)}[kind])
    if kind == "edges":  # the largest float below a power of two, with every low word; powers of two
        top = f32(1) - f32(2.0 ** -24)
        hi[::2] = np.where(rng.random(hi[::2].shape) < 0.5, top, -top)
        lo[::2] = rng.integers(-(2 ** 23), 2 ** 23 + 1, lo[::2].shape) * 2.0 ** -48
        hi[1::2] = 2.0 ** -rng.integers(1, 40, hi[1::2].shape)
        lo[1::2] = hi[1::2] * f32(2.0 ** -25) * rng.integers(-1, 2, hi[1::2].shape)
    E, d = _digits(lib, hi, lo, neg)
    assert np.all(np.abs(d[:, 0]) <= 256) and np.all(np.abs(d[:, 1:]) <= 128) and np.all(d == np.rint(d))
    for r in range(len(hi)):
        amax = float(np.abs(hi[r]).max())
        assert amax < 2.0 ** int(E[r]) and (amax == 0 or amax >= 2.0 ** (int(E[r]) - 1))
        for k in range(64):
            v = (Fraction(float(hi[r, k])) + Fraction(float(lo[r, k]))) / Fraction(2) ** int(E[r]) * (-1 if neg else 1)
            got = sum(Fraction(int(d[r, s, k])) / 2 ** (8 * (s + 1)) for s in range(7))
            # (the double-float value itself is rounded at 2^-69 while it is cut)
            assert abs(got - v) <= Fraction(1, 2 ** 57) + Fraction(1, 2 ** 68)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("other", [2.0 ** -140, 1e-30, 1.0, 1e30])
def test_rows_with_infinities_and_nan_give_no_finite_product(lib, bad, other):
    import torch
    hi = np.full((2, 64), other, f32)
    hi[0, 17] = bad
    lo = np.zeros_like(hi)
    E, _ = _digits(lib, hi, lo, False)
    assert E[0] == 1 << 20 and E[1] < 200
    e = torch.tensor([int(E[0] + E[1]) - 16], dtype=torch.int32, device="cuda")
    s = torch.zeros(1, device="cuda")
    assert lib.scale(1, device_kernels.ptr(e), device_kernels.ptr(s)) == 0
    # whatever the digits: a sum times this scale is infinite, or NaN where the sum is zero
    assert not np.isfinite(s.cpu().numpy()).any()


def test_folds_keep_the_group_sums(lib):
    import torch
    rng = np.random.default_rng(5)
    n = 4000
    top = np.array([2 ** 22, 2 ** 22, 5 * 2 ** 20, 6 * 2 ** 20, 7 * 2 ** 20, 8 * 2 ** 20, 9 * 2 ** 20])
    a = np.rint(rng.uniform(-1, 1, (n, 7)) * top * 10.0 ** rng.uniform(-7, 0, (n, 7)))
    a[:8] = top * (1 - 2 * (rng.random((8, 7)) < 0.5))
    a[8:200, 0] = 0                       # cancelling leading groups
    a[200:400, 1] = -256 * np.rint(a[200:400, 0] / 256)
    t = torch.tensor(a.astype(f32), device="cuda")
    out = torch.zeros(n, 4, device="cuda")
    assert lib.fold(n, device_kernels.ptr(t), device_kernels.ptr(out)) == 0
    o = out.cpu().numpy()
    bound = Fraction(4, 2 ** 24) + Fraction(2, 2 ** 32)
    for i in range(n):
        exact = sum(Fraction(int(a[i, u])) / 2 ** (8 * u) for u in range(7))
        for k in (0, 2):
            assert abs(Fraction(float(o[i, k])) + Fraction(float(o[i, k + 1])) - exact) <= bound
