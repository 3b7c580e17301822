"""Projected-gradient solves whose line search rejects most first steps (a large optimistic factor), so that a decision
often takes the values prepared for a rejection, on one cluster (up to 512 contacts) and on the grid: against the
oracle bit for bit, and the same in every repetition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nbodies", [(33, 11), (300, 100), (512, 200), (513, 200)])
@pytest.mark.parametrize("variant", [3, 1, 4])  # APGD, Descent, SPG (no line search: its momentum decisions)
def test_rejected_steps(oracle, n, nbodies, variant):
    import bogus_gpu
    from bogus_gpu import generator

    d = generator.random_pairs(nbodies, n, seed=300 + n)
    rp, cl, vl = oracle.PrimalProblem(d.minv, d.objA, d.objB, d.HA, d.HB).assemble()
    D = bogus_gpu.DualFrictionProblem()
    D.set(rp, cl, vl, d.b, d.mu)
    O = oracle.DualProblem(rp, cl, vl, d.b, d.mu)
    pg = bogus_gpu.ProjectedGradient()
    pg.setDefaultVariant(variant)
    pg.setTol(1e-13)
    pg.setMaxIters(150)
    pg.setLineSearchOptimisticFactor(5.0)
    pg.setLineSearchPessimisticFactor(0.4)
    for coulomb in (False, True):
        res_o, r_o, it_o = O.solve_pg(np.zeros(3 * n), variant=variant, coulomb=coulomb, tol=1e-13, max_iters=150,
                                      optimistic=5.0, pessimistic=0.4)
        for _ in range(5):
            r = np.zeros(3 * n)
            res = D.solveWith(pg, r, staticProblem=not coulomb)
            assert res == res_o and D.last_iterations == it_o and np.array_equal(r, r_o)
