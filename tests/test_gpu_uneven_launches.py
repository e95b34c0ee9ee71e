"""Uneven batches in the FP64 form: the mat-vec on small tiles runs for the columns
in which some matrix has 1 to 128 rows left, and no longer once the smallest matrix
has ended.  Cells of 28 and 148 atoms against two cells of 148 in one batch: the
only further launches are those of the smaller matrix's 83 columns."""
import numpy as np
import pytest

from parphom_gb300 import api, synth

pytestmark = pytest.mark.gpu


def test_no_empty_mat_vecs_after_the_smallest_matrix():
    cells = [synth.tblg_cell(1), synth.tblg_cell(3), synth.tblg_cell(3)]
    ctxs = [api.PhononContext.from_cell(c, synth.spring_force_constants(c, seed=0)) for c in cells]
    q = synth.random_qpoints(2, seed=7)
    o = api.EigOpts(jobz="N", precision=api.PP_PREC_FP64)
    count, out = [], []
    for which in ([2, 1], [0, 1]):
        before = api.kernel_launches()
        out.append(api.solve_multi(ctxs, np.array(which, dtype=np.int64), q, o, want_z=False))
        count.append(api.kernel_launches() - before)
    n = cells[0].n
    with ctxs[0] as c, ctxs[1], ctxs[2]:
        own = c.solve(q[:1], o)
    assert np.array_equal(out[0].w[1], out[1].w[1])   # (the second q-point, of a 148-atom cell both times)
    assert np.abs(out[1].w[0, :n] - own.w[0, :n]).max() <= 1e-9
    assert count[1] - count[0] == n - 1, count
