"""Calls whose memory does not hold the optional buffers (the factor's entries copied for the walked levels, the dense tail's
inverse): they run without them, with the same result to the solve's tolerance (relative residual 1e-8 on both sides).
SSP_WORKSPACE_LIMIT_MB stands for a smaller device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRAPHS = {
    "rgg": lambda ssp: ssp.gen_rgg(4000, 16.0, 0.1, 10.0, 5),
    "mesh": lambda ssp: ssp.gen_grid3d(14, 13, 12, -1.0, 1.0, 2),
}


def _prm(ssp, precision, k=70):
    p = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8)
    p.precision = precision
    p.jl_dim_override = k
    p.factor_max_degree = 0
    return p


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_runs_without_the_optional_buffers(ssp, monkeypatch, name, precision):
    G, prm = GRAPHS[name](ssp), _prm(ssp, precision)
    with ssp.Context(0) as c:
        H0, st0 = c.sparsify(G, prm)
        full = c.workspace_bytes
    # what the entries' copies alone take: 2 x 16 B an entry, 2 x 16 B a vertex (which of the optional buffers go is not said)
    extra = 32 * (st0["nnz_factor"] + G.n)
    monkeypatch.setenv("SSP_WORKSPACE_LIMIT_MB", str((full - extra) / 2**20))
    with ssp.Context(0) as c:
        for _ in range(2):
            H, st = c.sparsify(G, prm)
            assert c.workspace_bytes <= full - extra
            assert st["nnz_factor"] == st0["nnz_factor"] and st["m_out"] == st0["m_out"]
            assert st["pcg_max_relres"] < 1e-7 and abs(st["pcg_max_iters_used"] - st0["pcg_max_iters_used"]) <= 3
            assert np.array_equal(H.rowidx, H0.rowidx)
            np.testing.assert_allclose(H.values, H0.values, rtol=1e-6 if precision else 1e-8, atol=0)


@pytest.mark.parametrize("dense", [0, 4096])
def test_precond_matches_oracle_without_them(ssp, ora, monkeypatch, dense):
    """Every level launched, the dense tail's among them, to the bound of the walked form (n eps of the largest value)."""
    G = GRAPHS["rgg"](ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    cp, ri, va = ora.laplacian(G.n, v1, v2, w)
    L = ssp.CSC(G.n, cp, ri, va)
    R = np.random.default_rng(1).standard_normal((G.n, 40))
    o = ora.Factor(G.n, cp, ri, va, 11, dense, 0)
    Zo = np.column_stack([o.precond(R[:, j].copy()) for j in range(0, 40, 13)])
    with ssp.Context(0) as c:
        ssp.stage_precond(c, L, 11, R, dense, 0)
        full = c.workspace_bytes
    extra = 32 * (len(o.rows) + G.n)
    monkeypatch.setenv("SSP_WORKSPACE_LIMIT_MB", str((full - extra) / 2**20))
    with ssp.Context(0) as c:
        Z = ssp.stage_precond(c, L, 11, R, dense, 0)
    assert np.abs(Z[:, ::13] - Zo).max() <= 1e-12 * np.abs(Zo).max()


def test_too_little_memory_is_an_error_and_the_context_goes_on(ssp, monkeypatch):
    G, prm = GRAPHS["rgg"](ssp), _prm(ssp, 0)
    with ssp.Context(0) as c:
        H0, _ = c.sparsify(G, prm)
        c.release_workspace()
        monkeypatch.setenv("SSP_WORKSPACE_LIMIT_MB", "4")
        with pytest.raises(ssp.SspError, match="NOMEM"):
            c.sparsify(G, prm)
        monkeypatch.delenv("SSP_WORKSPACE_LIMIT_MB")
        H, _ = c.sparsify(G, prm)
    np.testing.assert_array_equal(H.values.view(np.uint64), H0.values.view(np.uint64))


def test_columns_in_batches_under_a_limit(ssp, monkeypatch):
    """Most of this graph's rows are cut into segments, whose sums count towards a batch's columns."""
    G = ssp.gen_er(1500, 600.0, 0.5, 2.0, 2)
    prm = _prm(ssp, 0, 600)
    prm.factor_max_degree = 640
    with ssp.Context(0) as c:
        H0, st0 = c.sparsify(G, prm)
        full = c.workspace_bytes
    block = 8 * G.n * 608
    monkeypatch.setenv("SSP_WORKSPACE_LIMIT_MB", str((full - 3 * block) / 2**20))
    with ssp.Context(0) as c:
        H, st = c.sparsify(G, prm)
        assert c.workspace_bytes <= full - 3 * block
    assert st["m_out"] == st0["m_out"] and np.array_equal(H.rowidx, H0.rowidx)
    np.testing.assert_allclose(H.values, H0.values, rtol=1e-8, atol=0)
