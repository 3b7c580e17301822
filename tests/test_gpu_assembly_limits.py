"""Delassus matrices with more blocks than an int counts are refused before anything is written, and the handle keeps
the dual problem it had."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [46341, 70000])  # one body in every contact: n^2 blocks, from the first size past 2^31 - 1
def test_too_many_blocks(oracle, n):
    import bogus_gpu
    from bogus_gpu import generator

    d = generator.random_pairs(24, 64, seed=2)
    small = bogus_gpu.PrimalFrictionProblem.from_generated(d)
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(small)
    pg = bogus_gpu.ProjectedGradient()
    pg.setMaxIters(50)
    r = np.zeros(3 * 64)
    res = D.solveWith(pg, r, staticProblem=True)

    H = np.zeros((n, 3, 1))
    H[:, 0, 0] = 1.0
    big = bogus_gpu.PrimalFrictionProblem(np.ones((1, 1, 1)), np.zeros(n, np.int32), np.full(n, -1, np.int32), H, np.zeros_like(H),
                                          np.zeros(3 * n), np.full(n, 0.5))
    with pytest.raises(bogus_gpu.BogusGpuError) as e:
        D.computeFrom(big)
    assert e.value.status == bogus_gpu.BAD_INPUT and "2^31" in str(e.value)

    again = np.zeros(3 * 64)
    assert D.solveWith(pg, again, staticProblem=True) == res and np.array_equal(again, r)
    D.computeFrom(small)
    again = np.zeros(3 * 64)
    assert D.solveWith(pg, again, staticProblem=True) == res and np.array_equal(again, r)
