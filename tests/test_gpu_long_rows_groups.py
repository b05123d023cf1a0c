"""Graphs most of whose Laplacian rows are cut into segments: the segments' sums are kept for some column tiles at a time, so
that they take at most half of one of the solve's n x k blocks, and a product is launched in groups of tiles.

Solutions have the residual asked for (recomputed with scipy in FP64: the tolerance plus 1 % for rounding), the diff norms
of the final product are those of the separate pass bit for bit, and a batch agrees with lone calls as batches do
(relative residual 1e-8 on both sides: 1e-8 in FP64, 0.5 % of the kept edges in mixed precision)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dense(ssp, n=1500, degree=600.0, seed=2):
    return ssp.gen_er(n, degree, 0.5, 2.0, seed)


def test_partial_sums_take_half_a_block_at_most(ssp):
    G = _dense(ssp, 3000, 1000.0)
    c = ssp.Context(0)
    try:
        L = ssp.stage_graph(c, G)[1]
        rng = np.random.default_rng(0)
        used = []
        for k in (32, 416):
            c.solve_lap(L, rng.standard_normal((G.n, k)), tol=1e-6, abs_tol=0.0, max_iters=100, max_degree=1100)
            used.append(c.workspace_bytes)
    finally:
        c.close()
    # per row and column: 3 blocks of the call and 5 of the PCG (64 B), half a block (4 B), and the reductions' partials of
    # at most 148 * 6 + 64 blocks three times over (8 B at this n)
    assert (used[1] - used[0]) / (384.0 * G.n) <= 64 + 4 + 8


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("k", [5, 33, 64, 200])
def test_solution_has_the_residual_asked_for(ssp, ctx, k, precision):
    G = _dense(ssp)
    L = ssp.stage_graph(ctx, G)[1]
    A = L.to_scipy()
    Y = np.random.default_rng(k).standard_normal((G.n, k))
    Z, rep = ctx.solve_lap(L, Y, tol=1e-9, abs_tol=0.0, max_iters=600, precision=precision)
    b = Y - Y.mean(0)
    rel = np.linalg.norm(b - A @ Z, axis=0) / np.linalg.norm(b, axis=0)
    assert rep["not_converged"] == 0 and rel.max() <= 1.01e-9


def test_diff_norms_of_the_final_product(ssp, ctx, monkeypatch):
    G = _dense(ssp)
    prm = ssp.SparsifierParameters.baseline(1.0, pcg_tol=1e-8)
    prm.jl_dim_override = 140
    prm.prob_variance_correction = 0  # small probabilities: the kept weights w / p show every bit of the norms
    H1, _ = ctx.sparsify(G, prm)
    monkeypatch.setenv("SSP_DIFF_FUSED", "0")
    H0, _ = ctx.sparsify(G, prm)
    np.testing.assert_array_equal(H1.rowidx, H0.rowidx)
    np.testing.assert_array_equal(H1.values.view(np.uint64), H0.values.view(np.uint64))


@pytest.mark.parametrize("precision", [0, 1])
def test_batch(ssp, ctx, precision):
    """Graphs of the batch stop at different iterations, so their rows are skipped tile by tile."""
    graphs = [_dense(ssp, 1000, 500.0, 1), ssp.gen_grid2d(30, 31), _dense(ssp, 1300, 400.0, 3)]
    params = []
    for i in range(3):
        p = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8, sampling_seed=i)
        p.dense_threshold = 0
        p.factor_max_degree = 24 if i == 1 else 0
        p.precision = precision
        p.jl_dim_override = 150 - 40 * i
        params.append(p)
    for G, p, (H, st) in zip(graphs, params, ctx.sparsify_batch(graphs, params)):
        H0, st0 = ctx.sparsify(G, p)
        assert st["pcg_max_relres"] < 1e-7
        if precision:
            assert abs(st["m_out"] - st0["m_out"]) <= 0.005 * st0["m_out"] + 1
        else:
            assert np.array_equal(H.rowidx, H0.rowidx)
            np.testing.assert_allclose(H.values, H0.values, rtol=1e-8, atol=0)
