"""The FP64 bisection's Sturm counts (the principal-minor recurrence with
rescaling) on tridiagonals where it can go wrong: exact zeros off the diagonal
and everywhere, clusters (Wilkinson's matrix, glued copies), graded entries,
minors that vanish at the bisection points, norms far from 1, orders around
the block of 8 rows.  Eigenvalues against LAPACK; the bound is the bisection's
own (2 ulp of the eigenvalue, or the abstol passed, one ulp of the norm: with 0
an eigenvalue that is exactly zero would need more halvings than there are)
plus a backward error of a few units in the last place of ||T|| from the
reduction and the counts."""
import numpy as np
import pytest

from parphom_gb300 import api

pytestmark = pytest.mark.gpu


def _cases():
    rng = np.random.default_rng(4)
    yield "zero", np.zeros(12), np.zeros(11)
    yield "equal", np.full(17, 3.0), np.zeros(16)
    yield "wilkinson", np.abs(np.arange(-10.0, 11.0)), np.ones(20)
    yield "glued", np.tile(np.abs(np.arange(-5.0, 6.0)), 9), np.tile(np.r_[np.ones(10), 1e-9], 9)[:-1]
    yield "half decoupled", rng.standard_normal(130), np.where(rng.random(129) < 0.5, 0.0, rng.standard_normal(129))
    yield "graded", 10.0 ** -np.arange(0, 30, 0.5), 0.3 * 10.0 ** -np.arange(0, 29.5, 0.5)
    yield "zero diagonal", np.zeros(65), np.ones(64)
    for n in (1, 2, 7, 8, 9, 10, 16, 17, 400):
        yield f"random {n}", rng.standard_normal(n), rng.standard_normal(n - 1)


@pytest.mark.parametrize("scale", [1.0, 1e-40, 1e40])
def test_fp64_bisection(scale):
    import torch
    dev = torch.device("cuda")
    for name, d, e in _cases():
        n = len(d)
        T = (np.diag(d) + np.diag(e, 1) + np.diag(e, -1)) * scale
        lam = np.linalg.eigvalsh(T)
        A = torch.tensor(T.astype(complex), device=dev)
        w = torch.zeros(n, dtype=torch.float64, device=dev)
        m = torch.zeros(1, dtype=torch.int64, device=dev)
        info = torch.zeros_like(m)
        rc = api.heevx_values_noalloc(A.data_ptr(), n, n, w.data_ptr(), m.data_ptr(), info.data_ptr(),
                                      abstol=2.0 ** -53 * float(np.abs(lam).max()))
        torch.cuda.synchronize()
        assert rc == 0 and int(m) == n and int(info) == 0, name
        norm = max(np.abs(lam).max(), 1e-300)
        err = np.abs(w.cpu().numpy() - lam).max()
        assert err <= (8 * n + 32) * 2.0 ** -53 * norm, (name, scale, err / norm)
