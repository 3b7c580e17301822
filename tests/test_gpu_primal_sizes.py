"""ADMM and DualAMA where their body phases split the work differently (bodies of 6 dofs), against the oracle exactly
equal (a crowded body's iterates may diverge: then NaN at the same places): bodies with no contact, one, and many, fewer bodies than a unit of
work and one past it, and both sides of the line between the kernels (a 32-contact chunk per warp of one CTA per SM)."""
import numpy as np
import pytest

import test_gpu_admm
import test_gpu_dual_ama

pytestmark = pytest.mark.gpu

LINE = 8 * 32 * 152


@pytest.fixture(scope="module")
def bg():
    import bogus_gpu

    bogus_gpu.lib()
    return bogus_gpu


def _data(n, nbodies, crowded):
    from bogus_gpu import generator

    d = (generator.random_pairs if n < 1000 else generator.grid)(nbodies, n, seed=n)
    objA, objB = np.array(d.objA), np.array(d.objB)
    if crowded:  # body 0 touches most contacts, the last body none
        objA[: n - n // 4] = 0
        objB[objB == 0] = -1
        objB[objB == nbodies - 1] = -1
        objA[objA == nbodies - 1] = 0
        objB[objB == objA] = -1
    HB = np.array(d.HB)
    return (d.minv, objA, objB, d.HA, HB, d.b, d.mu), nbodies


def _assert_same(g, o):
    for x, y in zip(g, o):
        assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True)


@pytest.mark.parametrize("n,nbodies,crowded,iters", [(1, 2, False, 40), (37, 5, True, 60), (61, 31, True, 60), (64, 33, False, 60),
                                                     (300, 97, False, 40), (LINE, 9000, False, 4), (LINE + 1, 9000, False, 4)])
def test_primal_sizes(bg, oracle, n, nbodies, crowded, iters):
    data, nb = _data(n, nbodies, crowded)
    rng = np.random.default_rng(n)
    f, v0, r0 = 0.1 * rng.standard_normal(6 * nb), 0.1 * rng.standard_normal(6 * nb), np.abs(0.01 * rng.standard_normal(3 * n))
    for lam in (0.0, 0.1):
        _assert_same(*test_gpu_admm._run_both(bg, oracle, data, lam, None, v0, r0, f, max_iters=iters))
    mass = np.linalg.inv(data[0])
    for ls in (0, 6):
        _assert_same(*test_gpu_dual_ama._run_both(bg, oracle, data, mass, f, v0, r0, ls=ls, max_iters=iters))
