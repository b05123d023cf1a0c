"""Streams that cannot hold the many-level launch of the factorization: it is refused, or its blocks give up waiting for one
another, and the levels are launched one by one, with the same factor bit for bit as the oracle's (example.cc:332-471)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WAYS = {"refused": ("SSP_FACTOR_LEVEL_BLOCKS", "100000"), "gives_up": ("SSP_FACTOR_LEVEL_SPINS", "0")}
CASES = {
    "grid": (lambda ssp: ssp.gen_grid2d(41, 40), 64, 0),
    "rgg": (lambda ssp: ssp.gen_rgg(3000, 16.0, 0.1, 10.0, 5), 0, 0),
    "truncated": (lambda ssp: ssp.gen_er(4000, 12.0, 0.5, 2.0, 2), 128, 16),
}


@pytest.mark.parametrize("way", list(WAYS))
@pytest.mark.parametrize("name", list(CASES))
def test_factor_matches_oracle(ssp, ora, ctx, monkeypatch, name, way):
    make, dense, maxdeg = CASES[name]
    G = make(ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    cp, ri, va = ora.laplacian(G.n, v1, v2, w)
    L = ssp.CSC(G.n, cp, ri, va)
    a = ctx.kernels_launched
    ssp.stage_factor(ctx, L, 5, dense, maxdeg)
    b = ctx.kernels_launched
    monkeypatch.setenv(*WAYS[way])
    f = ssp.stage_factor(ctx, L, 5, dense, maxdeg)
    c = ctx.kernels_launched
    o = ora.Factor(G.n, cp, ri, va, 5, dense, maxdeg)
    assert c - b > b - a  # several launches a level where one did many
    assert np.array_equal(f["level"], o.level)
    assert np.array_equal(f["D"].view(np.uint64), o.D.view(np.uint64))
    for v in range(G.n):
        p, q = slice(f["colptr"][v], f["colptr"][v + 1]), slice(o.colstart[v], o.colstart[v + 1])
        i, j = np.argsort(f["rows"][p]), np.argsort(o.rows[q])
        assert np.array_equal(f["rows"][p][i], o.rows[q][j])
        assert np.array_equal(f["vals"][p][i].view(np.uint64), o.vals[q][j].view(np.uint64))


@pytest.mark.parametrize("way", list(WAYS))
def test_batch_is_the_same(ssp, ctx, monkeypatch, way):
    graphs = [ssp.gen_grid2d(20, 21), ssp.gen_rgg(1200, 12.0, 0.1, 10.0, 3), ssp.gen_er(900, 40.0, 0.5, 2.0, 9)]
    params = []
    for i, deg in enumerate((0, 12, -1)):
        p = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8, sampling_seed=i)
        p.dense_threshold = 0
        p.factor_max_degree = deg
        params.append(p)
    want = ctx.sparsify_batch(graphs, params)
    monkeypatch.setenv(*WAYS[way])
    got = ctx.sparsify_batch(graphs, params)
    for (H, st), (H0, st0) in zip(got, want):
        assert st["nnz_factor"] == st0["nnz_factor"] and st["factor_levels"] == st0["factor_levels"]
        assert np.array_equal(H.rowidx, H0.rowidx)
        np.testing.assert_array_equal(H.values.view(np.uint64), H0.values.view(np.uint64))


def test_stream_with_a_part_of_the_device(ssp, ctx):
    """A caller's stream that owns 16 SMs (a green context)."""
    cu = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1:] if len(r) > 2 else (r[1] if len(r) == 2 else None)

    dev = ok(cu.cuDeviceGet(0))
    sms = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 16))
    desc = ok(cu.cuDevResourceGenerateDesc(groups, 1))
    green = ok(cu.cuGreenCtxCreate(desc, dev, cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(cu.cuGreenCtxStreamCreate(green, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    G = ssp.gen_rgg(3000, 16.0, 0.1, 10.0, 5)
    L = ssp.stage_graph(ctx, G)[1]
    want = ssp.stage_factor(ctx, L, 5, 64, 0)
    c = ssp.Context(0)
    try:
        c.set_stream(int(stream))
        got = ssp.stage_factor(c, L, 5, 64, 0)
    finally:
        c.close()
        ok(cu.cuStreamDestroy(stream))
        ok(cu.cuGreenCtxDestroy(green))
    for key in ("level", "D", "colptr"):
        np.testing.assert_array_equal(got[key], want[key])
    assert np.sort(got["vals"]).tolist() == np.sort(want["vals"]).tolist()
