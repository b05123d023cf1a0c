"""The Laplacian product and the final product at row lengths around the segment size (256 entries).

A row of more than 256 entries is cut into segments that different warps sum; the result must solve the system to the
tolerance asked for (the residual is recomputed here in FP64 with scipy, so it is at most the tolerance plus rounding,
1 % is allowed for it), and the diff norms formed by the final product must be those of the separate pass bit for bit.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

# entries of the hub rows of the Laplacian, the diagonal among them
HUBS = [255, 256, 257, 511, 512, 513, 770]


def _hub_graph(ssp, n=900):
    rng = np.random.default_rng(1)
    rows, cols = [np.arange(n - 1)], [np.arange(1, n)]  # a path keeps it connected
    for h, entries in enumerate(HUBS):
        hub = n + h
        leaves = rng.choice(n, entries - 1, replace=False)
        rows.append(np.full(entries - 1, hub))
        cols.append(leaves)
    r, c = np.concatenate(rows), np.concatenate(cols)
    N = n + len(HUBS)
    A = sp.coo_matrix((rng.uniform(0.5, 2.0, len(r)), (r, c)), shape=(N, N))
    return ssp.CSC.from_scipy(A + A.T)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("k", [5, 8, 33])
def test_solution_has_the_residual_asked_for(ssp, ctx, k, precision):
    G = _hub_graph(ssp)
    L = ssp.stage_graph(ctx, G)[1]
    A = L.to_scipy()
    assert set(HUBS) <= set(np.diff(A.indptr))
    Y = np.random.default_rng(k).standard_normal((G.n, k))
    Z, rep = ctx.solve_lap(L, Y, tol=1e-9, abs_tol=0.0, max_iters=600, precision=precision)
    b = Y - Y.mean(0)
    rel = np.linalg.norm(b - A @ Z, axis=0) / np.linalg.norm(b, axis=0)
    assert rep["not_converged"] == 0 and rel.max() <= 1.01e-9


def test_diff_norms_of_the_final_product(ssp, ctx, monkeypatch):
    G = _hub_graph(ssp)
    prm = ssp.SparsifierParameters.baseline(1.0, pcg_tol=1e-8)
    prm.jl_dim_override = 45
    prm.prob_variance_correction = 0  # small probabilities: the kept weights w / p show every bit of the norms
    H1, _ = ctx.sparsify(G, prm)
    monkeypatch.setenv("SSP_DIFF_FUSED", "0")
    H0, _ = ctx.sparsify(G, prm)
    np.testing.assert_array_equal(H1.rowidx, H0.rowidx)
    np.testing.assert_array_equal(H1.values.view(np.uint64), H0.values.view(np.uint64))
