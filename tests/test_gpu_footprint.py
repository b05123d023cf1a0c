"""The serving layer's memory estimate against what a context holds after the call, where the factor's copies, the dense
tail's inverse and the long rows' partial sums count; and a request whose needs fit its budget but not all it would take."""
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "complete_with_tail": (lambda ssp: ssp.gen_rgg(4000, 16.0, 0.1, 10.0, 5), 0, 0),
    "complete_er": (lambda ssp: ssp.gen_er(4000, 14.0, 0.5, 2.0, 3), 0, 0),
    "mixed_mesh": (lambda ssp: ssp.gen_grid3d(20, 20, 20, -3.0, 3.0, 2), 0, 1),
    "long_rows": (lambda ssp: ssp.gen_er(3000, 1000.0, 0.5, 2.0, 3), 1100, 0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_estimate_covers_the_workspace(ssp, name):
    make, degree, precision = CASES[name]
    G = make(ssp)
    prm = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8)
    prm.factor_max_degree = degree
    prm.precision = precision
    with ssp.Context(0) as c:
        c.sparsify(G, prm)
        assert ssp.request_footprint(G, prm) >= c.workspace_bytes


def test_request_whose_needs_fit_is_served_alone(ssp):
    G = CASES["complete_with_tail"][0](ssp)
    prm = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8)
    ld = (prm.jl_dim(G.n) + 31) // 32 * 32
    T = min(G.n, prm.dense_threshold)
    besides = 180 * G.nnz + 32 * G.n + 8 * T * T + 8 * T * ld
    with ssp.Server(0, slots=2, hbm_budget_bytes=ssp.request_footprint(G, prm) - besides) as srv:
        res = [srv.wait(t) for t in [srv.submit(G, prm) for _ in range(2)]]
        info = srv.info()
    assert info["completed"] == 2 and info["peak_inflight"] == 1 and info["rejected"] == 0
    assert res[0][1]["m_out"] == res[1][1]["m_out"]
