"""Rounding of M^{-1} r against extended precision.

The dense tail is applied as the inverse of its triangular block: sums of up to T terms in place of a solve's short rows.
Such a sum is formed in chains of eight terms that are added up exactly, so that its rounding (eight additions and the last
one, about eps) is that of a row solved by itself, whatever T.  The yardstick is the oracle's sequential FP64 solve on the
same factor: its error and the device's are sums of the same kind in other orders, which differ by less than a factor of 2
over a whole application; a plain chain of T terms would round like sqrt(T / 8) times that, 4 to 13 times at these
tails of 128 to 1300 vertices.  The algebra is custom_cg.hpp:224-235's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRAPHS = {
    "er3k": lambda ssp: ssp.gen_er(3000, 20.0, 0.5, 2.0, 1),
    "er2k_dense": lambda ssp: ssp.gen_er(2000, 100.0, 0.5, 2.0, 1),
    "rmat12": lambda ssp: ssp.gen_rmat(12, 16, 0.57, 0.19, 0.19, 3),
    "mesh": lambda ssp: ssp.gen_grid3d(21, 20, 19, -3.0, 3.0, 2),
}


def _extended(o, r):
    """L^{-T} D^+ L^{-1} r in extended precision, column by column of L in the elimination's order."""
    LD = np.longdouble
    order = np.argsort(o.level, kind="stable")
    vals, D = o.vals.astype(LD), o.D.astype(LD)
    y = r.astype(LD)
    for v in order:
        a, b = o.colstart[v], o.colstart[v + 1]
        if b > a:
            y[o.rows[a:b]] -= vals[a:b, None] * y[v]
    y = np.where(D[:, None] != 0, y / np.where(D == 0, 1, D)[:, None], y)
    for v in order[::-1]:
        a, b = o.colstart[v], o.colstart[v + 1]
        if b > a:
            y[v] -= (vals[a:b, None] * y[o.rows[a:b]]).sum(0)
    return y


@pytest.mark.parametrize("k", [8, 40])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_tail_rounds_like_a_row_by_row_solve(ssp, ora, ctx, name, k):
    G = GRAPHS[name](ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    cp, ri, va = ora.laplacian(G.n, v1, v2, w)
    o = ora.Factor(G.n, cp, ri, va, 7, 4096, 0)
    R = np.random.default_rng(k).standard_normal((G.n, k))
    Z = ssp.stage_precond(ctx, ssp.CSC(G.n, cp, ri, va), 7, R, 4096, 0)
    cols = np.linspace(0, k - 1, 8).astype(int)
    X = _extended(o, R[:, cols])
    Zo = np.column_stack([o.precond(R[:, j].copy()) for j in cols])
    rms = [float(np.sqrt(((z - X) ** 2).mean())) for z in (Z[:, cols], Zo)]
    assert rms[0] <= 2.0 * rms[1]
