"""The double-float multiply-adds as the device computes them: sums of 16 complex
products, one lane's share of a mat-vec tile, in one accumulator of the exact-product
multiply-add and in the mat-vec's two sums of the shorter one.

Bound of both: that of the emulated 16-term real sums (4 x 2^-46 of sum |x y|),
doubled for the 32 real products of a component.  The mat-vec's sums must not be
less accurate than the one accumulator: their rms error over the cases against its
own (a numpy emulation of 40000 sums of each kind of input gives 0.50 to 0.65 of it;
0.9 leaves 8 standard errors of this test's 2000)."""
from fractions import Fraction

import numpy as np
import pytest

from tests import device_kernels

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_kernels.load("dfsum", tmp_path_factory.mktemp("dfsum"))


def _df(x):
    hi = x.astype(f32)
    return np.stack([hi, (x - hi.astype(np.float64)).astype(f32)], axis=-1)


@pytest.mark.parametrize("conj", [0, 1])
@pytest.mark.parametrize("spread,positive", [(0, False), (2, False), (6, False), (0, True)])
def test_tile_sums(lib, conj, spread, positive):
    import torch
    rng = np.random.default_rng(7 + spread)
    cases, n = 2000, 16
    x = [rng.standard_normal((cases, n)) * 10.0 ** rng.uniform(-spread, 0, (cases, n)) for _ in range(4)]
    if positive:
        x = [np.abs(v) for v in x]
    a, b = (np.stack([_df(x[k]), _df(x[k + 1])], axis=2).reshape(cases, n, 4).astype(f32) for k in (0, 2))
    dev = torch.device("cuda")
    A, B = torch.tensor(a, device=dev), torch.tensor(b, device=dev)
    one, two = torch.zeros(cases, 4, device=dev), torch.zeros(cases, 4, device=dev)
    p = device_kernels.ptr
    assert lib.sums(cases, conj, p(A), p(B), p(one), p(two)) == 0
    one, two = one.cpu().numpy(), two.cpu().numpy()
    err = np.zeros((2, 2, cases))

    def F(v):
        return Fraction(float(v))

    for c in range(cases):
        s, mag = [Fraction(0), Fraction(0)], [0.0, 0.0]
        for k in range(n):
            ar, ai = F(a[c, k, 0]) + F(a[c, k, 1]), F(a[c, k, 2]) + F(a[c, k, 3])
            br, bi = F(b[c, k, 0]) + F(b[c, k, 1]), F(b[c, k, 2]) + F(b[c, k, 3])
            ai = -ai if conj else ai
            s[0] += ar * br - ai * bi
            s[1] += ar * bi + ai * br
            mag[0] += float(abs(ar * br) + abs(ai * bi))
            mag[1] += float(abs(ar * bi) + abs(ai * br))
        for f, out in enumerate((one, two)):
            for h in range(2):
                err[f, h, c] = float(F(out[c, 2 * h]) + F(out[c, 2 * h + 1]) - s[h]) / mag[h] * 2.0 ** 46
    assert np.abs(err).max() < 2 * 4
    rms = np.sqrt((err ** 2).mean(axis=(1, 2)))
    assert rms[1] <= 0.9 * rms[0], rms
