"""The factor tuner's probe keeps its residual history on the device and runs its iterations without waiting for one.  On
tiny graphs every column stops within a few of them: the rest must change nothing, alone or beside a graph that does
not stop (the batch's own tolerance against a lone call, 1e-8)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 5, 12, 40])
def test_probe_past_convergence(ssp, ctx, n):
    G = ssp.CSC.from_scipy(sp.csc_matrix(1.5 * (np.ones((n, n)) - np.eye(n))))
    other = ssp.gen_grid2d(30, 31)
    prm = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8)
    prm.dense_threshold = 0
    prm.factor_max_degree = -1  # the tuner decides
    for g, (Hb, st) in zip((G, other), ctx.sparsify_batch([G, other], [prm, prm])):
        H, st0 = ctx.sparsify(g, prm)
        assert np.isfinite(H.values).all() and st["m_out"] == st0["m_out"]
        assert np.array_equal(Hb.colptr, H.colptr) and np.array_equal(Hb.rowidx, H.rowidx)
        np.testing.assert_allclose(Hb.values, H.values, rtol=1e-8, atol=0)
