"""Solves whose values overflow (finite inputs, infinities and NaN in the residuals) take the same branches in every CTA
that shares them: against the schedule with one CTA per problem, NaN for NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nbodies", [(5, 3), (33, 11), (64, 24), (200, 70), (512, 180), (600, 200)])
@pytest.mark.parametrize("every", [1, 5, 37])  # contacts whose velocity is out of range
def test_overflow(n, nbodies, every):
    import bogus_gpu
    from bogus_gpu import generator

    d = generator.random_pairs(nbodies, n, seed=n)
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(bogus_gpu.PrimalFrictionProblem.from_generated(d))
    rp, cl, vl = D.W_lower()
    for scale in (1e155, 1e200, 1e300):
        b = d.b.reshape(-1, 3).copy()
        b[::every] *= scale
        E = bogus_gpu.DualFrictionProblem()
        E.set(rp, cl, vl, b.reshape(-1), d.mu)
        E.setBatch(np.array([0, n], np.int32))
        E.setBatchShape(0, 1, 1)
        for variant in (3, 4, 1):
            for inf_norm in (True, False):
                pg = bogus_gpu.ProjectedGradient()
                pg.setDefaultVariant(variant)
                pg.setTol(1e-14)
                pg.setMaxIters(20)
                pg.useInfinityNorm(inf_norm)
                r, s = np.zeros(3 * n), np.zeros(3 * n)
                res = E.solveWith(pg, r, staticProblem=False)
                res_b, its = E.solveBatchWith(pg, s, staticProblem=False)
                assert np.array_equal([res], res_b, equal_nan=True) and E.last_iterations == its[0]
                assert np.array_equal(r, s, equal_nan=True), (scale, variant, inf_norm)
