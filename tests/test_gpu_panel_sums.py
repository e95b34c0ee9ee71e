"""The sum w^H v of a panel column and alpha = -1/2 tau (w^H v), in the device's
own functions: no less than an FP64 product and sum.

A lane's sum keeps products and sums as three floats: each of its K additions
and products is off by at most a few 2^-70 of the terms so far; taken as K 2^-64
of sum |w v|, which an FP64 sum does not reach.  alpha is one FP64 product of
that, rounded to double-float: 2^-51 of |tau| |w^H v| from two FP64 roundings and
2^-49 from the low word, 2^-48 in all, and 32 lanes' sums."""
from fractions import Fraction

import numpy as np
import pytest

from tests import device_kernels

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_kernels.load("sums", tmp_path_factory.mktemp("sums"))


def _df(x):
    hi = x.astype(f32)
    return np.stack([hi, (x - hi.astype(np.float64)).astype(f32)], axis=-1)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 200])
@pytest.mark.parametrize("spread", [0, 8])
def test_products_and_sums_keep_fp64_accuracy(lib, n, spread):
    import torch
    rng = np.random.default_rng(n + spread)
    cases = 12
    x = [rng.standard_normal((cases, n)) * 10.0 ** rng.uniform(-spread, 0, (cases, n)) for _ in range(4)]
    if n > 32:  # the last entries cancel the first to a few units in the last place
        for a in (0, 1):
            x[a][:6, 32] = -x[a][:6, 0]
            x[2 + a][:6, 32] = x[2 + a][:6, 0] * (1 + 2.0 ** -44)
    w = np.stack([_df(x[0]), _df(x[1])], axis=2).reshape(cases, n, 4).astype(f32)
    v = np.stack([_df(x[2]), _df(x[3])], axis=2).reshape(cases, n, 4).astype(f32)
    t = rng.standard_normal((cases, 2))
    dev = torch.device("cuda")
    W, V, T = (torch.tensor(a, device=dev) for a in (w, v, t))
    own, out = torch.zeros(cases, 32, 6, device=dev), torch.zeros(cases, 4, device=dev)
    p = device_kernels.ptr
    assert lib.sums(cases, n, p(W), p(V), p(T), p(own), p(out)) == 0
    own, out = own.cpu().numpy(), out.cpu().numpy()

    def F(a):
        return Fraction(float(a))

    for c in range(cases):
        tot, terms = [Fraction(0), Fraction(0)], Fraction(0)
        for lane in range(32):
            s, mag = [Fraction(0), Fraction(0)], Fraction(0)
            for k in range(lane, n, 32):
                wr, wi = F(w[c, k, 0]) + F(w[c, k, 1]), F(w[c, k, 2]) + F(w[c, k, 3])
                vr, vi = F(v[c, k, 0]) + F(v[c, k, 1]), F(v[c, k, 2]) + F(v[c, k, 3])
                s[0] += wr * vr + wi * vi
                s[1] += wr * vi - wi * vr
                mag += (abs(wr) + abs(wi)) * (abs(vr) + abs(vi))
            for h in range(2):
                got = sum(F(own[c, lane, 3 * h + k]) for k in range(3))
                assert abs(got - s[h]) <= (n // 32 + 1) * mag / 2 ** 64
                tot[h] += s[h]
            terms += mag
        tr, ti = F(t[c, 0]), F(t[c, 1])
        want = (-(tr * tot[0] - ti * tot[1]) / 2, -(tr * tot[1] + ti * tot[0]) / 2)
        size = (abs(tr) + abs(ti)) * (abs(tot[0]) + abs(tot[1])) / 2
        slack = (abs(tr) + abs(ti)) * terms * (n + 32) / 2 ** 64
        for h in range(2):
            assert abs(F(out[c, 2 * h]) + F(out[c, 2 * h + 1]) - want[h]) <= size / 2 ** 48 + slack
