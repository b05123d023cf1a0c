"""Column batches when the memory is less than expected: the blocks of an earlier call count as free for the next one, and the
next may need others (FP32 blocks beside them).  A batch that runs out of memory is taken again with fewer columns, with
the result of a call that had the room.  SSP_WORKSPACE_LIMIT_MB stands for the device's size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _prm(ssp, precision, k):
    p = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8)
    p.precision = precision
    p.jl_dim_override = k
    p.factor_max_degree = 22
    return p


def test_mixed_call_after_a_larger_fp64_one(ssp, monkeypatch):
    """The FP64 call's blocks leave no room for the FP32 ones, though the estimate takes them for free (its reserve of 1 GiB
    needs blocks of this size to fail)."""
    G = ssp.gen_er(150000, 20.0, 0.5, 2.0, 1)
    k = 1000
    with ssp.Context(0) as c:
        H0, st0 = c.sparsify(G, _prm(ssp, 1, k))
        c.release_workspace()
        c.sparsify(G, _prm(ssp, 0, k))
        fp64 = c.workspace_bytes
        monkeypatch.setenv("SSP_WORKSPACE_LIMIT_MB", str(fp64 / 2**20 + 300.0))
        H, st = c.sparsify(G, _prm(ssp, 1, k))
        assert c.workspace_bytes <= fp64 + 300 * 2**20
    assert st["m_out"] == st0["m_out"] and st["pcg_max_relres"] < 1e-7
    assert np.array_equal(H.rowidx, H0.rowidx)
    np.testing.assert_allclose(H.values, H0.values, rtol=1e-6, atol=0)


@pytest.mark.parametrize("precision", [0, 1])
def test_all_columns_at_once_take_more_than_expected(ssp, monkeypatch, precision):
    """A factor far denser than the graph leaves less than the estimate made before it sets aside."""
    G = ssp.gen_er(12000, 14.0, 0.5, 2.0, 3)
    p = _prm(ssp, precision, 500)
    p.factor_max_degree = 0
    with ssp.Context(0) as c:
        H0, st0 = c.sparsify(G, p)
        full = c.workspace_bytes
    optional = 32 * (st0["nnz_factor"] + G.n) + 8 * 4096 * 4096  # the copies, and at most this for the dense tail's inverse
    block = 8 * G.n * 512
    monkeypatch.setenv("SSP_WORKSPACE_LIMIT_MB", str((full - optional - 2 * block) / 2**20))
    with ssp.Context(0) as c:
        H, st = c.sparsify(G, p)
    assert st["m_out"] == st0["m_out"] and st["pcg_max_relres"] < 1e-7
    assert np.array_equal(H.rowidx, H0.rowidx)
    np.testing.assert_allclose(H.values, H0.values, rtol=1e-6 if precision else 1e-8, atol=0)
