"""The triangular solves' walked levels and dense tails against the oracle.

Levels are walked inside one launch by blocks of 8 columns (clusters of blocks where the columns leave SMs idle, smaller
blocks where there are many columns), and the one-vertex-per-level tail of complete elimination is applied as the
inverse of its triangular block.  Both only reorder each row's sum, so M^{-1} r must agree with the oracle's sequential
solve to 1e-12 of its largest value: row sums of at most n terms of one sign round by about n eps = 1e-13 relative,
and the tail's inverse has entries in [0, 1].  The preconditioner's algebra is custom_cg.hpp:224-235's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star(ssp, n):
    """A hub with n - 1 leaves, the leaves joined in a path: one row of L holds about n entries."""
    import scipy.sparse as sp
    i = np.arange(1, n)
    r = np.concatenate([np.zeros(n - 1, int), i[:-1]])
    c = np.concatenate([i, i[1:]])
    A = sp.coo_matrix((np.random.default_rng(4).uniform(0.5, 2.0, len(r)), (r, c)), shape=(n, n))
    return ssp.CSC.from_scipy(A + A.T)


def _path(ssp, n):
    import scipy.sparse as sp
    i = np.arange(n - 1)
    A = sp.coo_matrix((np.ones(n - 1), (i, i + 1)), shape=(n, n))
    return ssp.CSC.from_scipy(A + A.T)


GRAPHS = {
    "grid31x29": lambda ssp: ssp.gen_grid2d(31, 29),
    "grid3d_9": lambda ssp: ssp.gen_grid3d(9, 9, 9, -3, 3, 2),
    "star1500": lambda ssp: _star(ssp, 1500),
    "path65": lambda ssp: _path(ssp, 65),
    "pair": lambda ssp: _path(ssp, 2),
    "rgg700": lambda ssp: ssp.gen_rgg(700, 14.0, 0.1, 10.0, 3),
}


# columns: the narrow layout (8), clusters of 8, 4 and 2 blocks, one block of 1024 threads, blocks of 512 and 256
@pytest.mark.parametrize("k", [1, 8, 9, 33, 64, 200, 500, 1185, 2400])
@pytest.mark.parametrize("name,dense", [("grid31x29", 4096), ("grid31x29", 0), ("grid3d_9", 4096), ("star1500", 4096),
                                        ("star1500", 0), ("path65", 4096), ("path65", 0), ("pair", 4096), ("pair", 0),
                                        ("rgg700", 4096), ("rgg700", 0)])
def test_precond_matches_oracle(ssp, ora, ctx, name, dense, k):
    G = GRAPHS[name](ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    cp, ri, va = ora.laplacian(G.n, v1, v2, w)
    R = np.random.default_rng(k).standard_normal((G.n, k))
    Z = ssp.stage_precond(ctx, ssp.CSC(G.n, cp, ri, va), 11, R, dense, 0)
    o = ora.Factor(G.n, cp, ri, va, 11, dense, 0)
    cols = sorted({0, 1, 7, 8, 31, 32, k // 2, k - 2, k - 1} & set(range(k)))
    Zo = np.column_stack([o.precond(R[:, j].copy()) for j in cols])
    assert np.abs(Z[:, cols] - Zo).max() <= 1e-12 * np.abs(Zo).max()


@pytest.mark.parametrize("name", ["grid31x29", "rgg700"])
def test_precond_is_the_same_in_every_run(ssp, ora, ctx, name):
    """The storage order is fixed by the factor (level, length, id), so repeated calls give the same bits."""
    G = GRAPHS[name](ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    L = ssp.CSC(G.n, *ora.laplacian(G.n, v1, v2, w))
    R = np.random.default_rng(0).standard_normal((G.n, 70))
    Z = [ssp.stage_precond(ctx, L, 5, R, 4096, 0) for _ in range(3)]
    for z in Z[1:]:
        np.testing.assert_array_equal(z.view(np.uint64), Z[0].view(np.uint64))
