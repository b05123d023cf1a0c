"""The truncation's diagonal takes its second launch, blocks for bags of more than 32 entries, only where there is such a
bag.  Two circulant graphs truncated before their first level differ in nothing else."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _circulant(ssp, n, d):
    r = np.concatenate([np.arange(n) for _ in range(d // 2)])
    c = np.concatenate([(np.arange(n) + j + 1) % n for j in range(d // 2)])
    A = sp.coo_matrix((np.random.default_rng(d).uniform(0.5, 2.0, len(r)), (r, c)), shape=(n, n)).tocsr()
    return ssp.CSC.from_scipy(A + A.T)


def test_block_launch_only_for_large_bags(ssp, ora, ctx):
    launches = []
    for d in (32, 34):
        G = _circulant(ssp, 400, d)
        v1, v2, w = ora.extract_edges(G.n, G.colptr, G.rowidx, G.values)
        L = ssp.CSC(G.n, *ora.laplacian(G.n, v1, v2, w))
        a = ctx.kernels_launched
        f = ssp.stage_factor(ctx, L, 9, 0, d - 1)
        launches.append(ctx.kernels_launched - a)
        assert len(f["rows"]) == 0 and f["level"].max() == 0
    assert launches[1] == launches[0] + 2  # stage_factor runs twice
