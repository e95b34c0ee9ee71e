"""The tensor-core tile update (trailing update of the reduction and X -= V Y of
the back-transform) where its split changes: one row past a 128-row block, odd
numbers of 64-column blocks, and batches that give a CTA one, two and four
column blocks, on random cells without any structure.

Residual and orthogonality of all eigenpairs in the mixed form, in float64 on
the matrix the library assembles; bounds of the other vector tests
(1e-11 ||D|| and 1e-10)."""
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


@pytest.mark.parametrize("natom,nq", [(11, 2), (22, 3), (43, 3), (54, 40), (65, 3), (86, 90), (97, 12), (129, 1),
                                      (129, 12), (129, 60)])
def test_eigenpairs_over_column_block_splits(natom, nq):
    lat, pos, phi = _random_cell(natom, natom)
    crys = geometry.crys_from_positions(lat, pos)
    rng = np.random.default_rng(nq)
    qs = np.concatenate([rng.uniform(-0.5, 0.5, (nq, 2)), np.zeros((nq, 1))], axis=1)
    n = 3 * natom
    with api.PhononContext(lat, crys, pos, np.array([1.0]), np.ones(natom, np.int64), phi) as ctx:
        r = ctx.solve(qs, api.EigOpts(jobz="V", precision=api.PP_PREC_MIXED, raw_lambda=True))
        for t in sorted({0, nq // 2, nq - 1}):
            D = ctx.dynamical_matrix(qs[t])
            D = np.triu(D) + np.triu(D, 1).conj().T
            norm = np.linalg.norm(D, 2)
            Z, lam = r.z[t][:, :n], r.w[t, :n]
            assert r.m[t] == n and r.nz[t] == n and r.info[t] == 0
            assert np.linalg.norm(D @ Z - Z * lam, axis=0).max() <= 1e-11 * norm
            assert np.abs(Z.conj().T @ Z - np.eye(n)).max() <= 1e-10


@pytest.mark.parametrize("natom", [1, 11, 21, 22, 43, 64, 65, 86])
def test_velocities_without_and_with_vectors(natom):
    """The product X^H Z of the velocities without eigenvectors, at chunks of 64
    rows, tiles of 128 eigenvectors and their remainders, against the velocities
    formed from the eigenvectors of the same tridiagonal problem.  v w is linear
    in products of vector pairs that differ by the two transforms' rounding, at
    most about sqrt(n) 2^-44 each with ||dD/dq|| = max |v w| up to a small factor:
    64 sqrt(n) 2^-44."""
    lat, pos, phi = _random_cell(natom, natom)
    crys = geometry.crys_from_positions(lat, pos)
    qs = np.array([[0.11, 0.23, 0.0], [0.37, -0.19, 0.0]])
    n = 3 * natom
    with api.PhononContext(lat, crys, pos, np.array([1.0]), np.ones(natom, np.int64), phi) as ctx:
        a = ctx.solve(qs, api.EigOpts(jobz="N", vel=True, precision=api.PP_PREC_MIXED), want_z=False)
        z = ctx.solve(qs, api.EigOpts(jobz="V", vel=True, precision=api.PP_PREC_MIXED))
        for t in range(len(qs)):
            va, vz = (r.vel[t, :n] * np.abs(r.w[t, :n, None]) for r in (a, z))
            assert np.isfinite(va).all()
            assert np.abs(va - vz).max() <= 64 * np.sqrt(n) * 2.0 ** -44 * np.abs(vz).max()
