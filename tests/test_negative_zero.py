"""A friction coefficient of -0.0 is one of 0.0: per-contact functions and whole solves against the oracle, bit for bit,
and against the same input with +0.0."""
import numpy as np
import pytest


def test_law_functions(oracle, hostmath):
    rng = np.random.default_rng(5)
    points = [np.array([-1.0, 0.3, 0.4]), np.array([1.0, 0.3, 0.4]), np.array([0.0, 0.3, 0.4]), np.array([-0.0, 0.0, 0.5]),
              np.zeros(3), np.array([-1.0, 0.0, 0.0]), np.array([-1.0, -0.0, 0.0]), np.array([2.0, 0.0, -0.0])]
    points += list(rng.standard_normal((500, 3)))
    A = np.array([[2.0, 0.3, -0.2], [0.3, 1.5, 0.1], [-0.2, 0.1, 1.2]]).reshape(-1)
    for x in points:
        p, q = x.copy(), x.copy()
        hostmath.hm_project(-0.0, p)
        hostmath.hm_project(0.0, q)
        assert np.array_equal(p, oracle.project(-0.0, x)) and np.array_equal(p, q)
        for coulomb in (False, True):
            y = rng.standard_normal(3)
            e = hostmath.hm_law_eval(int(coulomb), -0.0, x, y)
            assert e == oracle.law_eval(-0.0, x, y, coulomb) == hostmath.hm_law_eval(int(coulomb), 0.0, x, y)
            for strategy in range(4):
                out = []
                for mu in (-0.0, 0.0):
                    v = x.copy()
                    res = hostmath.hm_local_solve(int(coulomb), strategy, A, y, v, mu, 1.8189894035458565e-12, 1.0)
                    out.append((res, v))
                res_o, x_o = oracle.local_solve(A.reshape(3, 3), y, x, -0.0, coulomb=coulomb, strategy=strategy, scaling=1.0)
                assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
                assert np.array_equal(out[0][1], x_o)


@pytest.mark.gpu
@pytest.mark.parametrize("n,nbodies", [(70, 24), (700, 300), (6000, 2000)])
def test_solves(oracle, n, nbodies):
    import bogus_gpu
    from bogus_gpu import generator

    d = generator.random_pairs(nbodies, n, seed=9)
    mu = d.mu.copy()
    mu[::3] = -0.0
    rp, cl, vl = oracle.PrimalProblem(d.minv, d.objA, d.objB, d.HA, d.HB).assemble()
    b = d.b.copy()
    b.reshape(-1, 3)[::6, 0] = np.abs(b.reshape(-1, 3)[::6, 0]) + 1.0  # separating: an attracting force would not vanish
    O = oracle.DualProblem(rp, cl, vl, b, mu)
    D, P = bogus_gpu.DualFrictionProblem(), bogus_gpu.DualFrictionProblem()
    D.set(rp, cl, vl, b, mu)
    P.set(rp, cl, vl, b, np.where(mu == 0, 0.0, mu))
    r0 = np.random.default_rng(n).standard_normal(3 * n)
    for variant in (3, 4, 1):
        for coulomb in (False, True):
            pg = bogus_gpu.ProjectedGradient()
            pg.setDefaultVariant(variant)
            pg.setTol(1e-10)
            pg.setMaxIters(40)
            res_o, r_o, it_o = O.solve_pg(r0, variant=variant, coulomb=coulomb, tol=1e-10, max_iters=40)
            for E in (D, P):
                r = r0.copy()
                assert E.solveWith(pg, r, staticProblem=not coulomb) == res_o
                assert E.last_iterations == it_o and np.array_equal(r, r_o)
    gs = bogus_gpu.GaussSeidel()
    gs.setMaxIters(20)
    gs.setTol(1e-12)
    out = []
    for E in (D, P):
        r = r0.copy()
        out.append((E.solveWith(gs, r), r))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
    # FP32-refined: both parts agree on the sign
    pg = bogus_gpu.ProjectedGradient()
    pg.setTol(1e-10)
    pg.setMaxIters(40)
    pg.setMixedPrecision(True, 20)
    out = []
    for E in (D, P):
        r = r0.copy()
        out.append((E.solveWith(pg, r, staticProblem=True), r))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
