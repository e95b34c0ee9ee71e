"""Linear triangulation at the sizes where its kernel splits the work (32
triangles per warp, 32 energies at a time, 512 energies per block) and at values
that tie: energies on vertices, equal vertices, energies in no order, against
the oracle.  Tolerances of the other triangulation tests."""
import numpy as np
import pytest

from oracle import dos_ref
from parphom_gb300 import dos

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,nb,ntri,ne,ties", [(3, 1, 1, 1, False), (3, 1, 1, 33, True), (16, 3, 31, 32, True),
                                                (16, 3, 32, 100, False), (16, 2, 33, 511, True), (25, 1, 65, 512, False),
                                                (25, 1, 40, 513, True), (36, 2, 70, 1030, True)])
def test_triangulation_edges(nk, nb, ntri, ne, ties):
    rng = np.random.default_rng(nk + ne)
    freq = rng.uniform(-3, 20, (nk, nb))
    E = rng.uniform(-5, 22, ne)
    if ties:
        freq, E = np.round(freq), np.round(2 * E) / 2
    func = rng.uniform(0.5, 1.5, freq.shape)
    tri = np.stack([rng.permutation(nk)[:3] for _ in range(ntri)]).astype(np.int64)
    d, n = dos.linear_triangulation(freq, tri, E, func)
    d_ref, n_ref = (np.asarray(a) for a in dos_ref.linear_triangulation(freq, func, tri, E))
    finite = np.isfinite(d_ref) & np.isfinite(n_ref)
    assert np.array_equal(np.isfinite(d) & np.isfinite(n), finite)
    for a, b in ((d, d_ref), (n, n_ref)):
        np.testing.assert_allclose(a[finite], b[finite], rtol=1e-10, atol=1e-12 * np.abs(b[finite]).max(initial=1.0))
