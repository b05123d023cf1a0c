"""Levels eliminated inside one launch against the oracle, bit for bit: bags at the edges of the warp tier (32), of the
counted sort (256) and of what the launch takes (512), with the levels before and after such a bag in either path, and
truncations on the way.  The elimination is example.cc:332-471's."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _circulant(ssp, n, d, seed):
    r = np.concatenate([np.arange(n) for _ in range(d // 2)])
    c = np.concatenate([(np.arange(n) + j + 1) % n for j in range(d // 2)])
    A = sp.coo_matrix((np.random.default_rng(seed).uniform(0.5, 2.0, len(r)), (r, c)), shape=(n, n)).tocsr()
    return ssp.CSC.from_scipy(A + A.T)


def _star(ssp, n, seed):
    r = np.zeros(n - 1, np.int64)
    A = sp.coo_matrix((np.random.default_rng(seed).uniform(0.5, 2.0, n - 1), (r, np.arange(1, n))), shape=(n, n)).tocsr()
    return ssp.CSC.from_scipy(A + A.T)


CASES = [(f"circulant_{n}_{d}_{dense}", lambda ssp, n=n, d=d: _circulant(ssp, n, d, n + d), dense, 0)
         for n, d, dense in ((3, 2, 0), (33, 2, 0), (300, 32, 0), (300, 34, 16), (600, 254, 0), (600, 258, 0),
                             (1300, 510, 64), (1300, 514, 64), (6000, 4, 0), (9001, 6, 128))] + \
        [("star", lambda ssp: _star(ssp, 5000, 1), 0, 0)] + \
        [("truncated", lambda ssp: _circulant(ssp, 5000, 8, 7), 128, 12)]


@pytest.mark.parametrize("name,make,dense,maxdeg", CASES, ids=[c[0] for c in CASES])
def test_levels_match_oracle(ssp, ora, ctx, name, make, dense, maxdeg):
    G = make(ssp)
    v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
    cp, ri, va = ora.laplacian(G.n, v1, v2, w)
    f = ssp.stage_factor(ctx, ssp.CSC(G.n, cp, ri, va), 5, dense, maxdeg)
    o = ora.Factor(G.n, cp, ri, va, 5, dense, maxdeg)
    assert np.array_equal(f["level"], o.level)
    assert np.array_equal(f["D"].view(np.uint64), o.D.view(np.uint64))
    of = np.repeat(np.arange(G.n), np.diff(f["colptr"]))
    oo = np.repeat(np.arange(G.n), np.diff(o.colstart))
    i, j = np.lexsort((f["rows"], of)), np.lexsort((o.rows[:len(oo)], oo))
    assert np.array_equal(f["rows"][i], o.rows[j])
    assert np.array_equal(f["vals"][i].view(np.uint64), o.vals[j].view(np.uint64))
