"""The forms of the triangular solves, each by itself: walked levels with clusters of 1, 2, 4 and 8 blocks, and every level
launched at 8, 16 and 32 columns per warp row.  Which of them a solve takes depends on its size, so the switches
SSP_TRSV_WALK, SSP_TRSV_CLUSTER and SSP_TRSV_WIDTH set them, and the solver's own report says what ran.

M^{-1} r agrees with the oracle's sequential solve to 1e-12 of its largest value (row sums of at most n terms round by about
n eps); launched levels agree bit for bit at every width.  FP32 solves precondition as well as FP64 ones: their rounding,
1e-7, against the 1e-8 asked of the FP64 iteration around them costs at most a few iterations (3 allowed).  The algebra
is custom_cg.hpp:224-235's."""
import re

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import rand_graph

pytestmark = pytest.mark.gpu


def _star(ssp, n):
    i = np.arange(1, n)
    r = np.concatenate([np.zeros(n - 1, int), i[:-1]])
    c = np.concatenate([i, i[1:]])
    A = sp.coo_matrix((np.random.default_rng(4).uniform(0.5, 2.0, len(r)), (r, c)), shape=(n, n))
    return ssp.CSC.from_scipy(A + A.T)


GRAPHS = {
    "grid3d": lambda ssp: ssp.gen_grid3d(12, 11, 10, -3, 3, 2),
    "rgg": lambda ssp: ssp.gen_rgg(3000, 14.0, 0.1, 10.0, 3),
    "star": lambda ssp: _star(ssp, 1500),  # a row of about n entries
    "er_dense": lambda ssp: ssp.CSC.from_scipy(rand_graph(1500, 110_000, 5)),  # rows longer than a chunk
    "rmat": lambda ssp: ssp.gen_rmat(11, 16, 0.57, 0.19, 0.19, 3),
}


def _lap(ssp, ora, name):
    G = GRAPHS[name](ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    return G.n, ssp.CSC(G.n, *ora.laplacian(G.n, v1, v2, w))


def _report(ssp, ctx, capfd, L, k, precision=0, dense=0, **kw):
    """(levels walked, columns a block, cluster, levels launched, tail) of one solve, and its report"""
    capfd.readouterr()
    Y = np.random.default_rng(5).standard_normal((L.n, k))
    _, rep = ctx.solve_lap(L, Y, tol=1e-8, abs_tol=0.0, max_iters=400, factor_seed=11, dense_threshold=dense, max_degree=0,
                           precision=precision, verbose=True, **kw)
    m = re.findall(r"triangular solves( \(fp32\))?: (\d+) levels walked \((\d+) columns, \d+ threads, clusters of (\d+)\), "
                   r"(\d+) launched, dense tail of (\d+)", capfd.readouterr().err)
    assert len(m) >= 1 and (m[0][0] != "") == (precision != 0 and k > 8)
    return tuple(int(x) for x in m[0][1:]), rep


@pytest.mark.parametrize("cl", [1, 2, 4, 8])
@pytest.mark.parametrize("k", [8, 33, 64])
@pytest.mark.parametrize("name,dense", [("grid3d", 0), ("grid3d", 4096), ("rgg", 0), ("rgg", 4096), ("star", 0),
                                        ("er_dense", 0)])
def test_walked_levels_match_oracle(ssp, ora, ctx, capfd, monkeypatch, name, dense, k, cl):
    n, L = _lap(ssp, ora, name)
    monkeypatch.setenv("SSP_TRSV_WALK", "1")
    monkeypatch.setenv("SSP_TRSV_CLUSTER", str(cl))
    (walked, cols, clusters, launched, tail), _ = _report(ssp, ctx, capfd, L, k, dense=dense)
    # the last level and the tail's earlier entries aside, every level of both directions
    assert walked > 0 and launched <= 2 and clusters == cl and cols == (2 if k <= 8 else 8)
    assert (tail > 0) == (dense > 0)
    R = np.random.default_rng(k).standard_normal((n, k))
    o = ora.Factor(n, L.colptr, L.rowidx, L.values, 11, dense, 0)
    Z = ssp.stage_precond(ctx, L, 11, R, dense, 0)
    js = sorted({0, 1, 7, k // 2, k - 1})
    Zo = np.column_stack([o.precond(R[:, j].copy()) for j in js])
    assert np.abs(Z[:, js] - Zo).max() <= 1e-12 * np.abs(Zo).max()


@pytest.mark.parametrize("walk", ["0", "1"])
@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("name,dense", [("grid3d", 0), ("grid3d", 4096), ("rgg", 4096), ("er_dense", 0), ("rmat", 4096)])
def test_fp32_forms_precondition_like_fp64(ssp, ora, ctx, capfd, monkeypatch, name, dense, precision, walk):
    n, L = _lap(ssp, ora, name)
    _, r64 = _report(ssp, ctx, capfd, L, 40, dense=dense)
    monkeypatch.setenv("SSP_TRSV_WALK", walk)
    monkeypatch.setenv("SSP_TRSV_CLUSTER", "4")
    (walked, _, _, launched, tail), rep = _report(ssp, ctx, capfd, L, 40, precision=precision, dense=dense)
    assert (walked == 0) == (walk == "0") and (launched > 2) == (walk == "0") and (tail > 0) == (dense > 0)
    assert rep["not_converged"] == 0
    if precision == 2:
        assert rep["max_iters_used"] <= r64["max_iters_used"] + 3


@pytest.mark.parametrize("name,maxdeg", [("er_dense", 0), ("er_dense", 200), ("rmat", 0), ("rmat", 40), ("grid3d", 0),
                                         ("rgg", 0)])
def test_launched_levels_of_every_width(ssp, ora, ctx, capfd, monkeypatch, name, maxdeg):
    n, L = _lap(ssp, ora, name)
    monkeypatch.setenv("SSP_TRSV_WALK", "0")
    R = np.random.default_rng(3).standard_normal((n, 40))
    out, counts = {}, {}
    for w in (8, 16, 32):
        monkeypatch.setenv("SSP_TRSV_WIDTH", str(w))
        (walked, _, _, launched, _), rep = _report(ssp, ctx, capfd, L, 40)
        per_width = {x: rep[f"trsv_levels_w{x}"] for x in (8, 16, 32)}
        assert walked == 0 and per_width[w] == sum(per_width.values()) > 2
        counts[w] = per_width[w]
        out[w] = ssp.stage_precond(ctx, L, 11, R, 0, maxdeg)
    assert len(set(counts.values())) == 1
    for w in (16, 32):
        np.testing.assert_array_equal(out[w].view(np.uint64), out[8].view(np.uint64), err_msg=f"width {w}")
    o = ora.Factor(n, L.colptr, L.rowidx, L.values, 11, 0, maxdeg)
    js = [0, 17, 39]
    Zo = np.column_stack([o.precond(R[:, j].copy()) for j in js])
    assert np.abs(out[8][:, js] - Zo).max() <= 1e-12 * np.abs(Zo).max()


@pytest.mark.parametrize("maxdeg", [0, 24])
def test_fp32_launched_widths_agree(ssp, monkeypatch, maxdeg):
    G = ssp.gen_er(6000, 14.0, 0.5, 2.0, 4)
    prm = ssp.SparsifierParameters.baseline(0.7, pcg_tol=1e-8)
    prm.precision = ssp.SSP_PRECISION_MIXED
    prm.jl_dim_override = 45
    prm.factor_max_degree = maxdeg
    prm.dense_threshold = 0
    monkeypatch.setenv("SSP_TRSV_WALK", "0")
    out = []
    for w in ("8", "16", "32"):
        monkeypatch.setenv("SSP_TRSV_WIDTH", w)
        with ssp.Context(0) as c:
            H, st = c.sparsify(G, prm)
        assert st[f"trsv_levels_w{w}"] == sum(st[f"trsv_levels_w{x}"] for x in (8, 16, 32)) > (2 if maxdeg == 0 else 0)
        out.append(H)
    for H in out[1:]:
        np.testing.assert_array_equal(H.rowidx, out[0].rowidx)
        np.testing.assert_array_equal(H.values.view(np.uint64), out[0].values.view(np.uint64))
