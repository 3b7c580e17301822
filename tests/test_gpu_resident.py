"""The projected-gradient kernel of problems that fit the SMs' shared memory (kernels_pg_resident.cu) at the sizes where
its split changes, against the oracle bit for bit (no tolerance: every value goes through the oracle's operations in
the oracle's order): a chunk per SM and one more, two to five teams per CTA with ragged last chunks, the last size that
fits and the first that does not, and rows long enough for the general kernel (more than 64 steps per lane)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SM = 152  # GB300


def _pair(oracle, n, nbodies, seed):
    import bogus_gpu
    from bogus_gpu import generator

    d = (generator.random_pairs if n < 1000 else generator.grid)(nbodies, n, seed=seed)
    rp, cl, vl = oracle.PrimalProblem(d.minv, d.objA, d.objB, d.HA, d.HB).assemble()
    D = bogus_gpu.DualFrictionProblem()
    D.set(rp, cl, vl, d.b, d.mu)
    return D, oracle.DualProblem(rp, cl, vl, d.b, d.mu)


def _compare(D, O, n, variant, coulomb, inf_norm, iters, r0):
    import bogus_gpu

    pg = bogus_gpu.ProjectedGradient()
    pg.setDefaultVariant(variant)
    pg.setMaxIters(iters)
    pg.setTol(1e-9)
    pg.useInfinityNorm(inf_norm)
    trace = []
    pg.callback().connect(lambda it, res: trace.append((it, res)))
    r = r0.copy()
    res = D.solveWith(pg, r, staticProblem=not coulomb)
    res_o, r_o, it_o = O.solve_pg(r0, variant=variant, coulomb=coulomb, tol=1e-9, max_iters=iters, inf_norm=inf_norm)
    assert res == res_o and D.last_iterations == it_o and np.array_equal(r, r_o), (variant, coulomb, inf_norm)
    assert len(trace) >= it_o


@pytest.mark.parametrize("n,nbodies", [(1, 2), (63, 3), (64, 24), (70, 4), (500, 200)])
def test_small(oracle, n, nbodies):
    D, O = _pair(oracle, n, nbodies, 40 + n)
    warm = np.abs(np.random.default_rng(n).standard_normal(3 * n))
    for variant in (3, 4, 1):  # APGD, SPG, Descent
        for coulomb in (False, True):
            for inf_norm in (False, True):
                _compare(D, O, n, variant, coulomb, inf_norm, 120, warm if coulomb else np.zeros(3 * n))


@pytest.mark.parametrize("n", [32 * SM - 5, 32 * SM + 1, 64 * SM + 17, 4 * 32 * SM - 1, 5 * 32 * SM, 5 * 32 * SM + 1])
def test_teams(oracle, n):
    D, O = _pair(oracle, n, n // 3, 7)
    for variant, coulomb in ((3, False), (4, True)):
        _compare(D, O, n, variant, coulomb, False, 15, np.zeros(3 * n))
