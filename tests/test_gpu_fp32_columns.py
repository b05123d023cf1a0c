"""FP32 products and solves with a lane holding two columns: row lengths around the gathers in flight, column counts that
end inside a pair, and level launches of every width.

A mixed-precision solve asks 1e-4 of each FP32 round, so 1e-9 takes three; one more is allowed for rounding.  A wrong entry
anywhere would cost rounds, or send them to FP64, before it cost accuracy.  The widths form each row in one order, so
their results agree bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _mixed_rows(ssp, n=1200):
    """A cycle with hubs of 2 .. 66 neighbours, so that Laplacian rows have 3 .. 67 entries."""
    rng = np.random.default_rng(2)
    rows, cols = [np.arange(n)], [(np.arange(n) + 1) % n]
    for h in range(65):
        rows.append(np.full(h + 2, n + h))
        cols.append(rng.choice(n, h + 2, replace=False))
    r, c = np.concatenate(rows), np.concatenate(cols)
    A = sp.coo_matrix((rng.uniform(0.5, 2.0, len(r)), (r, c)), shape=(n + 65, n + 65))
    return ssp.CSC.from_scipy(A + A.T)


@pytest.mark.parametrize("k", [9, 31, 32, 33, 34, 63])
def test_fp32_rounds_contract(ssp, ctx, k):
    G = _mixed_rows(ssp)
    L = ssp.stage_graph(ctx, G)[1]
    A = L.to_scipy()
    Y = np.random.default_rng(k).standard_normal((G.n, k))
    Z, rep = ctx.solve_lap(L, Y, tol=1e-9, abs_tol=0.0, max_iters=600, precision=1)
    b = Y - Y.mean(0)
    rel = np.linalg.norm(b - A @ Z, axis=0) / np.linalg.norm(b, axis=0)
    assert rep["not_converged"] == 0 and rel.max() <= 1.01e-9
    assert rep["fp64_rounds"] == 0 and rep["refinements"] <= 4


@pytest.mark.parametrize("maxdeg", [0, 24])
def test_fp32_level_widths_agree(ssp, monkeypatch, maxdeg):
    G = ssp.gen_er(6000, 14.0, 0.5, 2.0, 4)
    prm = ssp.SparsifierParameters.baseline(0.7, pcg_tol=1e-8)
    prm.precision = ssp.SSP_PRECISION_MIXED
    prm.jl_dim_override = 45
    prm.factor_max_degree = maxdeg
    prm.dense_threshold = 0
    out = []
    for w in ("8", "16", "32"):
        monkeypatch.setenv("SSP_TRSV_WIDTH", w)
        c = ssp.Context(0)
        try:
            out.append(c.sparsify(G, prm)[0])
        finally:
            c.close()
    for H in out[1:]:
        np.testing.assert_array_equal(H.rowidx, out[0].rowidx)
        np.testing.assert_array_equal(H.values.view(np.uint64), out[0].values.view(np.uint64))
