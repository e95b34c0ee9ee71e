"""Captured launch sequences that a context keeps: velocities mode by mode while
force constants change under them, and that tuning one configuration leaves
the others' alone.

Velocities: a call of a context that has replayed other sequences, with other
force constants (same non-zero blocks, other values; sparser; denser again), against
a context of its own.  Both solve D(q) with a backward error of at most tol ||D||
(tol of the eigenvalue tests), so a mode with gap g to its neighbours turns by at
most 2 tol ||D|| / g each, and v w, quadratic in the vector, changes by at most
16 tol ||D|| / g of the largest |v w| times a factor of 4 between that and the norm of
dD/dq.  Modes closer than 1e-6 ||D|| are left out; a block too few or misplaced
changes v w by much more than the 1e-4 this leaves."""
import time

import numpy as np
import pytest

from parphom_gb300 import api, geometry, synth

pytestmark = pytest.mark.gpu


def _cell(natom, seed, zero):
    rng = np.random.default_rng(seed)
    lat = np.array([[9.0, 0.0, 0.0], [4.5, 7.8, 0.0], [0.0, 0.0, 20.0]])
    pos = np.random.default_rng(1).random((natom, 3)) @ lat
    a = rng.standard_normal((natom, 3, natom, 3))
    keep = np.triu(np.random.default_rng(2).random((natom, natom)) > zero, 1)
    a *= (keep | keep.T | np.eye(natom, dtype=bool))[:, None, :, None]
    a = a.reshape(3 * natom, 3 * natom)
    return lat, pos, (a + a.T) / np.sqrt(6 * natom)


@pytest.mark.parametrize("prec", [api.PP_PREC_FP64, api.PP_PREC_MIXED])
def test_velocities_mode_by_mode(prec):
    natom, n = 24, 72
    rng = np.random.default_rng(3)
    qs = np.concatenate([rng.uniform(-0.4, 0.4, (6, 2)), np.zeros((6, 1))], axis=1)
    calls = [("N", 6), ("V", 4), ("N", 3), ("V", 6), ("N", 1), ("N", 6)]
    phis = [_cell(natom, 5, 0.4), _cell(natom, 6, 0.4), _cell(natom, 7, 0.8), _cell(natom, 8, 0.8), _cell(natom, 5, 0.4)]
    lat, pos, phi0 = phis[0]
    crys = geometry.crys_from_positions(lat, pos)
    mass, types = np.array([1.0]), np.ones(natom, np.int64)
    tol = 8 * n * 2.0 ** -53 if prec == api.PP_PREC_FP64 else (8 + 4 * np.sqrt(n)) * 2.0 ** -44
    compared = 0
    with api.PhononContext(lat, crys, pos, mass, types, phi0) as ctx:
        for k, (_, _, phi) in enumerate(phis):
            if k:
                ctx.update_fc(phi)
            for jobz, nq in calls:
                o = api.EigOpts(jobz=jobz, vel=True, precision=prec)
                r = ctx.solve(qs[:nq], o, want_z=jobz == "V")
                with api.PhononContext(lat, crys, pos, mass, types, phi) as own:
                    e = own.solve(qs[:nq], o, want_z=jobz == "V")
                for t in range(nq):
                    lam = np.sign(e.w[t, :n]) * e.w[t, :n] ** 2
                    norm = np.abs(lam).max()
                    gap = np.minimum(np.diff(lam, prepend=-np.inf), np.diff(lam, append=np.inf)) / norm
                    vr, ve = (x.vel[t, :n] * np.abs(x.w[t, :n, None]) for x in (r, e))
                    ok = gap > 1e-6
                    bound = 64 * tol / gap * np.abs(ve).max()
                    assert np.all(np.abs(vr - ve).max(axis=1)[ok] <= bound[ok]), (k, jobz, nq, t)
                    assert np.abs(ve).max() > 0
                    compared += ok.sum()
    assert compared > 0.95 * len(phis) * sum(nq for _, nq in calls) * n


def test_tuning_leaves_other_configurations_captured():
    """A captured configuration's pass takes as long after two others have been tuned (five captures each) as before;
    with a capture of its own it takes about twice that."""
    c = synth.tblg_cell(5)                                     # n = 1092
    phi = synth.spring_force_constants(c, seed=0)
    q = synth.random_qpoints(16, seed=5)

    def once(ctx, il, nq):
        o = api.EigOpts(jobz="N", range="I", il=il, iu=il + 3, precision=api.PP_PREC_MIXED)
        t = time.perf_counter()
        ctx.solve(q[:nq], o)
        return time.perf_counter() - t

    with api.PhononContext.from_cell(c, phi) as ctx:
        ctx.solve(q, api.EigOpts(jobz="N", precision=api.PP_PREC_MIXED))    # (sizes the workspace)
        once(ctx, 1, 16)
        before = min(once(ctx, 1, 16) for _ in range(3))
        after = []
        for nq in (15, 13, 11):                # (the best of three: a host may be busy once)
            once(ctx, 1, nq)
            once(ctx, 1, nq - 1)
            after.append(once(ctx, 1, 16))
    assert min(after) <= 1.3 * before, (before, after)
