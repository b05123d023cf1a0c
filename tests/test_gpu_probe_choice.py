"""The factor tuner's choice on graphs that its probe solves long before its last iteration.  What follows convergence are
rounding errors; the choice must not depend on them, so every sketch of such a graph keeps the light factor."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [False, True])
def test_converged_probe_keeps_the_light_factor(ssp, ctx, batched):
    G = ssp.gen_er(8000, 600.0, 0.5, 2.0, 1)
    for seed in range(4):
        prm = ssp.SparsifierParameters.baseline(0.5, pcg_tol=1e-8, sketch_seed=seed)
        prm.jl_dim_override = 64
        if batched:
            prm.dense_threshold = 0
            st = ctx.sparsify_batch([G], [prm])[0][1]
        else:
            st = ctx.sparsify(G, prm)[1]
        assert st["factor_max_degree_used"] > 0
        assert st["pcg_max_iters_used"] < 20
