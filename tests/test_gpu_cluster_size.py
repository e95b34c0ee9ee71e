"""The column step with smaller clusters than the device allows, as on a partition
that cannot place 16 CTAs together: the same eigenvalues, residuals and
orthogonality, at orders on both sides of the row kernel's threshold (512 rows)
and past the rows a cluster's shared memory holds (512 a CTA).

The sums are only dealt differently: the double-float form's keep 2^-66, so its
eigenvalues differ by the bisection's width (4 x 2^-44 ||T||), those of the FP64 form by
the reduction's rounding, n 2^-50 ||D|| as in the tests of the reduction."""
import numpy as np
import pytest

from parphom_gb300 import api, geometry

pytestmark = pytest.mark.gpu


def _cell(natom):
    rng = np.random.default_rng(natom)
    lat = np.array([[9.0, 0.0, 0.0], [4.5, 7.8, 0.0], [0.0, 0.0, 20.0]])
    pos = rng.random((natom, 3)) @ lat
    a = rng.standard_normal((3 * natom, 3 * natom))
    return lat, pos, (a + a.T) / np.sqrt(6 * natom)


@pytest.mark.parametrize("prec", [api.PP_PREC_FP64, api.PP_PREC_MIXED])
@pytest.mark.parametrize("natom", [2, 22, 86, 171, 203])
def test_smaller_clusters(natom, prec, monkeypatch):
    lat, pos, phi = _cell(natom)
    crys = geometry.crys_from_positions(lat, pos)
    n = 3 * natom
    qs = np.array([[0.11, 0.23, 0.0], [0.37, -0.19, 0.0]])
    res = {}
    for cap in (16, 8, 2, 1):
        monkeypatch.setenv("PARPHOM_GPU_CLUSTER", str(cap))
        with api.PhononContext(lat, crys, pos, np.array([1.0]), np.ones(natom, np.int64), phi) as ctx:
            r = ctx.solve(qs, api.EigOpts(jobz="V", precision=prec, raw_lambda=True))
            D = [ctx.dynamical_matrix(q) for q in qs]
        assert np.all(r.info == 0) and np.all(r.m == n)
        res[cap] = r.w[:, :n]
        for t in range(len(qs)):
            H = np.triu(D[t]) + np.triu(D[t], 1).conj().T
            norm = np.linalg.norm(H, 2)
            Z, lam = r.z[t][:, :n], r.w[t, :n]
            assert np.linalg.norm(H @ Z - Z * lam, axis=0).max() <= 1e-11 * norm
            assert np.abs(Z.conj().T @ Z - np.eye(n)).max() <= 1e-10
    scale = np.abs(res[16]).max()
    tol = n * 2.0 ** -50 if prec == api.PP_PREC_FP64 else (8 + 4 * np.sqrt(n)) * 2.0 ** -44
    for cap in (8, 2, 1):
        assert np.abs(res[cap] - res[16]).max() <= tol * scale
