"""A Gauss-Seidel sweep whose waits run out reports it and leaves the handle usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_timeout_then_solve(oracle):
    import bogus_gpu
    from bogus_gpu import generator

    L = bogus_gpu.lib()
    n = 501
    d = generator.random_pairs(200, n, seed=12)
    rp, cl, vl = oracle.PrimalProblem(d.minv, d.objA, d.objB, d.HA, d.HB).assemble()
    D = bogus_gpu.DualFrictionProblem()
    D.set(rp, cl, vl, d.b, d.mu)
    gs = bogus_gpu.GaussSeidel()
    gs.setMaxIters(50)
    gs.setTol(1e-14)
    gs.coloring().update(False)
    r = np.full(3 * n, 0.25)
    try:
        assert L.bogus_gpu_set_wait_limit(0, 1e-6) == bogus_gpu.OK  # below a local solve: some wait runs out
        with pytest.raises(bogus_gpu.BogusGpuError) as e:
            D.solveWith(gs, r)
        assert e.value.status == bogus_gpu.TIMEOUT and (r == 0.25).all()
    finally:
        assert L.bogus_gpu_set_wait_limit(0, 4.0) == bogus_gpu.OK
    r = np.zeros(3 * n)
    res = D.solveWith(gs, r)
    res_o, r_o, it_o = oracle.DualProblem(rp, cl, vl, d.b, d.mu).solve_gs(np.zeros(3 * n), coulomb=True, tol=1e-14, max_iters=50,
                                                                         coloring=False)
    assert res == res_o and D.last_iterations == it_o and np.array_equal(r, r_o)
