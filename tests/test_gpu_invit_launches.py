"""Inverse iteration in several launches that share their scratch: a thread does
the same work whatever launch it is in, so the vectors are those of one launch, bit
for bit -- with a last launch of few threads, with clusters (equal and nearly equal
eigenvalues) across the launches, and in a batch.  And the workspace of a large
batch does not grow by a thread per eigenvector."""
import numpy as np
import pytest

from parphom_gb300 import api, geometry, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [api.PP_PREC_FP64, api.PP_PREC_MIXED])
@pytest.mark.parametrize("natom,clustered", [(22, False), (75, False), (75, True)])
def test_launches_share_scratch(natom, clustered, prec, monkeypatch):
    rng = np.random.default_rng(natom)
    n = 3 * natom
    lat = np.array([[9.0, 0.0, 0.0], [4.5, 7.8, 0.0], [0.0, 0.0, 20.0]])
    pos = rng.random((natom, 3)) @ lat
    if clustered:  # every eigenvalue of Phi six times, and pairs 1e-9 apart
        Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        lam = np.repeat(rng.uniform(0.5, 2.0, n // 6 + 1), 6)[:n] * (1 + 1e-9 * (np.arange(n) % 2))
        phi = (Q * lam) @ Q.T
        phi = (phi + phi.T) / 2
        qs = np.zeros((2, 3))
    else:
        a = rng.standard_normal((n, n))
        phi = (a + a.T) / np.sqrt(2 * n)
        qs = np.array([[0.11, 0.23, 0.0], [0.37, -0.19, 0.0]])
    crys = geometry.crys_from_positions(lat, pos)
    monkeypatch.setenv("PARPHOM_GPU_TUNE", "0")
    out = {}
    for cap in ("0", "64", "32"):
        monkeypatch.setenv("PARPHOM_GPU_INVIT_THREADS", cap)
        with api.PhononContext(lat, crys, pos, np.array([1.0]), np.ones(natom, np.int64), phi) as ctx:
            out[cap] = ctx.solve(qs, api.EigOpts(jobz="V", precision=prec, raw_lambda=True))
    for cap in ("64", "32"):
        assert np.array_equal(out[cap].info, out["0"].info)
        assert np.array_equal(out[cap].w, out["0"].w)
        assert np.array_equal(out[cap].z, out["0"].z)


@pytest.mark.parametrize("nq,all_at_once", [(3, True), (24, False)])
def test_scratch_of_a_large_batch_is_bounded(nq, all_at_once, monkeypatch):
    """n = 2604: a thread per eigenvector (576 x 33 n bytes a matrix more) for 3 matrices, not for 24."""
    import torch
    c = synth.tblg_cell(8)
    phi = synth.spring_force_constants(c, seed=0)
    q = synth.random_qpoints(nq, seed=3)
    monkeypatch.setenv("PARPHOM_GPU_TUNE", "0")
    monkeypatch.setenv("PARPHOM_GPU_GRAPHS", "0")
    used = []
    for cap in ("0", "2048"):
        monkeypatch.setenv("PARPHOM_GPU_INVIT_THREADS", cap)
        with api.PhononContext.from_cell(c, phi) as ctx:
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            ctx.solve(q, api.EigOpts(jobz="N", vel=True, precision=api.PP_PREC_MIXED), want_z=False)
            used.append(free - torch.cuda.mem_get_info()[0])
    more = nq * 576 * 33 * c.n if all_at_once else 0
    assert abs(used[0] - used[1] - more) <= 1 << 26     # (allocations are rounded to 2 MB)
