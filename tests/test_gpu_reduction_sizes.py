"""The reduction at the orders where its kernels change shape: one and few
rows, the cluster sizes of the column step (a CTA per 8 rows up to 16), the
mat-vec's tiles (32 x 32 and 64 x 32), the panel width, and the order at which
the row work moves to a kernel of its own (512 rows), on random cells without
any structure, both precision forms, three q-points per batch.

Eigenvalues of D(q) against LAPACK on the matrix the library assembles.  The
bound: a backward-stable reduction to an order-n tridiagonal perturbs an
eigenvalue by at most a modest multiple of n eps ||D||, eps = 2^-53, resp. the
double-float unit 2^-47 with errors that add up like sqrt(n) over the rows
(taken as n^(1/2) 2^-44 with the bisection's own stopping width 4 * 2^-44)."""
import numpy as np
import pytest

from parphom_gb300 import api, geometry

pytestmark = pytest.mark.gpu


def _random_cell(natom, seed):
    rng = np.random.default_rng(seed)
    lat = np.array([[9.0, 0.0, 0.0], [4.5, 7.8, 0.0], [0.0, 0.0, 20.0]])
    pos = rng.random((natom, 3)) @ lat
    a = rng.standard_normal((3 * natom, 3 * natom))
    phi = (a + a.T) / np.sqrt(6 * natom)
    return lat, pos, phi


@pytest.mark.parametrize("prec", [api.PP_PREC_FP64, api.PP_PREC_MIXED])
@pytest.mark.parametrize("natom", [1, 2, 3, 5, 6, 11, 21, 22, 32, 43, 54, 86, 171, 172, 182, 203])
def test_eigenvalues_at_edge_orders(natom, prec):
    lat, pos, phi = _random_cell(natom, natom)
    crys = geometry.crys_from_positions(lat, pos)
    qs = np.array([[0.11, 0.23, 0.0], [0.37, -0.19, 0.0], [-0.28, 0.41, 0.0]])
    n = 3 * natom
    with api.PhononContext(lat, crys, pos, np.array([1.0]), np.ones(natom, np.int64), phi) as ctx:
        r = ctx.solve(qs, api.EigOpts(jobz="N", precision=prec, raw_lambda=True))
        for t, q in enumerate(qs):
            D = ctx.dynamical_matrix(q)
            D = np.triu(D) + np.triu(D, 1).conj().T
            lam = np.linalg.eigvalsh(D)
            norm = np.abs(lam).max()
            tol = 8 * n * 2.0 ** -53 if prec == api.PP_PREC_FP64 else (8 + 4 * np.sqrt(n)) * 2.0 ** -44
            assert r.m[t] == n and r.info[t] == 0
            assert np.abs(r.w[t, :n] - lam).max() <= tol * norm, (n, np.abs(r.w[t, :n] - lam).max() / norm)
