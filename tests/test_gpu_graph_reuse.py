"""Calls of one context that alternate between more configurations than it keeps
captured launch sequences for, with force constants replaced in between (same
and different non-zero blocks): every call as from a context of its own.  The
two differ by rounding at most (the launch configuration is chosen per call);
bounds of the eigenvalue tests."""
import numpy as np
import pytest

from parphom_gb300 import api, geometry

pytestmark = pytest.mark.gpu


def _cell(natom, seed, zero):
    rng = np.random.default_rng(seed)
    lat = np.array([[9.0, 0.0, 0.0], [4.5, 7.8, 0.0], [0.0, 0.0, 20.0]])
    pos = np.random.default_rng(1).random((natom, 3)) @ lat
    a = rng.standard_normal((natom, 3, natom, 3))
    keep = np.random.default_rng(2).random((natom, natom)) > zero
    a *= (keep & keep.T)[:, None, :, None]
    a = a.reshape(3 * natom, 3 * natom)
    return lat, pos, (a + a.T) / np.sqrt(6 * natom)


@pytest.mark.parametrize("prec", [api.PP_PREC_FP64, api.PP_PREC_MIXED])
def test_alternating_configurations_and_force_constants(prec):
    natom, n = 24, 72
    rng = np.random.default_rng(3)
    qs = np.concatenate([rng.uniform(-0.4, 0.4, (7, 2)), np.zeros((7, 1))], axis=1)
    calls = [("N", 7), ("V", 4), ("N", 3), ("V", 7), ("N", 1), ("V", 4), ("N", 7)]
    phis = [_cell(natom, 5, 0.4), _cell(natom, 6, 0.4), _cell(natom, 7, 0.9), _cell(natom, 5, 0.4)]
    lat, pos, phi0 = phis[0]
    crys = geometry.crys_from_positions(lat, pos)
    mass, types = np.array([1.0]), np.ones(natom, np.int64)
    with api.PhononContext(lat, crys, pos, mass, types, phi0) as ctx:
        for k, (_, _, phi) in enumerate(phis):
            if k:
                ctx.update_fc(phi)
            for jobz, nq in calls:
                o = api.EigOpts(jobz=jobz, vel=jobz == "N", precision=prec, raw_lambda=True)
                r = ctx.solve(qs[:nq], o, want_z=jobz == "V")
                with api.PhononContext(lat, crys, pos, mass, types, phi) as own:
                    e = own.solve(qs[:nq], o, want_z=jobz == "V")
                norm = np.abs(e.w).max()
                tol = 8 * n * 2.0 ** -53 if prec == api.PP_PREC_FP64 else (8 + 4 * np.sqrt(n)) * 2.0 ** -44
                assert np.abs(r.w - e.w).max() <= 2 * tol * norm
                if jobz == "N":
                    assert np.abs(r.vel).max() <= 2 * np.abs(e.vel).max() and np.abs(e.vel).max() <= 2 * np.abs(r.vel).max()
                else:
                    for t in range(nq):
                        D = ctx.dynamical_matrix(qs[t])
                        D = np.triu(D) + np.triu(D, 1).conj().T
                        Z = r.z[t][:, :n]
                        assert np.linalg.norm(D @ Z - Z * r.w[t, :n], axis=0).max() <= 1e-11 * norm
