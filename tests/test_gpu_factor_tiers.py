"""The factor's size tiers against the oracle, bit for bit: the truncation's diagonal (a warp up to 32 live entries, a
block above) and the dense tail's columns (ranked by counting up to 512 nonzeros, sorted by the network above).  The
elimination is example.cc:332-471's."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import rand_graph

pytestmark = pytest.mark.gpu


def _complete(ssp, n):
    A = np.triu(np.random.default_rng(n).uniform(0.5, 2.0, (n, n)), 1)
    return ssp.CSC.from_scipy(sp.csc_matrix(A + A.T))


def _regular(ssp, n, d):
    """A circulant graph: every vertex has d neighbours, so the first truncation sees bags of about d entries."""
    r = np.concatenate([np.arange(n) for _ in range(d // 2)])
    c = np.concatenate([(np.arange(n) + j + 1) % n for j in range(d // 2)])
    A = sp.coo_matrix((np.random.default_rng(d).uniform(0.5, 2.0, len(r)), (r, c)), shape=(n, n)).tocsr()
    return ssp.CSC.from_scipy(A + A.T)


CASES = [(f"regular{d}", lambda ssp, d=d: _regular(ssp, 400, d), 4096, d - 1) for d in (30, 32, 34, 66)] + \
        [("er_mixed_bags", lambda ssp: ssp.CSC.from_scipy(rand_graph(900, 14_000, 3)), 0, 33)] + \
        [(f"complete{n}", lambda ssp, n=n: _complete(ssp, n), 4096, 0) for n in (2, 33, 34, 512, 513, 514, 700)]


@pytest.mark.parametrize("name,make,dense,maxdeg", CASES, ids=[c[0] for c in CASES])
def test_factor_matches_oracle(ssp, ora, ctx, name, make, dense, maxdeg):
    G = make(ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    cp, ri, va = ora.laplacian(G.n, v1, v2, w)
    f = ssp.stage_factor(ctx, ssp.CSC(G.n, cp, ri, va), 9, dense, maxdeg)
    o = ora.Factor(G.n, cp, ri, va, 9, dense, maxdeg)
    assert np.array_equal(f["level"], o.level)
    assert np.array_equal(f["D"].view(np.uint64), o.D.view(np.uint64))
    for v in range(G.n):  # a column's entries, whatever order they are stored in
        a = slice(f["colptr"][v], f["colptr"][v + 1])
        b = slice(o.colstart[v], o.colstart[v + 1])
        i, j = np.argsort(f["rows"][a]), np.argsort(o.rows[b])
        assert np.array_equal(f["rows"][a][i], o.rows[b][j])
        assert np.array_equal(f["vals"][a][i].view(np.uint64), o.vals[b][j].view(np.uint64))
