"""Chunks cut on the device: windows of 256 rows, chunks of at most 32 rows and 256 entries, longer rows cut into segments.
A row left out or taken twice would not survive the residual, recomputed here in FP64 (1 % allowed for its rounding)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _graph(ssp, n, deg, hubs, seed=1):
    rng = np.random.default_rng(seed)
    r, c = [np.arange(n - 1)], [np.arange(1, n)]
    if deg:
        m = n * deg // 2
        a, b = rng.integers(0, n, m), rng.integers(0, n, m)
        r.append(a[a != b])
        c.append(b[a != b])
    for h in hubs:  # rows whose windows hold a long row: first, last and inside
        leaves = rng.choice(n, 300, replace=False)
        leaves = leaves[leaves != h]
        r.append(np.full(len(leaves), h))
        c.append(leaves)
    r, c = np.concatenate(r), np.concatenate(c)
    A = sp.coo_matrix((rng.uniform(0.5, 2.0, len(r)), (r, c)), shape=(n, n)).tocsr()
    return ssp.CSC.from_scipy(A + A.T)


CASES = [(2, 0, ()), (255, 0, ()), (256, 0, ()), (257, 3, ()), (513, 40, (0, 255, 256, 512)), (2048, 6, (2047,)),
         (2049, 6, ()), (9000, 12, (17, 8192))]


@pytest.mark.parametrize("maxdeg", [0, 4])
@pytest.mark.parametrize("n,deg,hubs", CASES)
def test_residual(ssp, ctx, n, deg, hubs, maxdeg):
    G = _graph(ssp, n, deg, hubs)
    L = ssp.stage_graph(ctx, G)[1]
    A = L.to_scipy()
    Y = np.random.default_rng(n).standard_normal((n, 9))
    Z, rep = ctx.solve_lap(L, Y, tol=1e-9, abs_tol=0.0, max_iters=4000, max_degree=maxdeg)
    b = Y - Y.mean(0)
    rel = np.linalg.norm(b - A @ Z, axis=0) / np.linalg.norm(b, axis=0)
    assert rep["not_converged"] == 0 and rel.max() <= 1.01e-9
