"""Delassus assembly of scenes in which a body is in many contacts (terrain as a body): against the oracle bit for bit, and
in a time that grows with the blocks and not with their number per row squared."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub(n, hubs, seed):
    """n contacts, each of one of `hubs` bodies with one of its own (every 11th with the other hub)."""
    rng = np.random.default_rng(seed)
    objA = (np.arange(n) % hubs).astype(np.int32)
    objB = (hubs + np.arange(n)).astype(np.int32)
    if hubs > 1:
        objB[::11] = (objA[::11] + 1) % hubs
    nb = hubs + n
    HA, HB = rng.standard_normal((2, n, 3, 6))
    R = rng.standard_normal((nb, 6, 6))
    return np.einsum("bij,bkj->bik", R, R) + np.eye(6), objA, objB, HA, HB, rng.standard_normal(3 * n), np.full(n, 0.5)


@pytest.mark.parametrize("n,hubs", [(600, 1), (1025, 2)])
def test_hub(oracle, n, hubs):
    import bogus_gpu

    minv, objA, objB, HA, HB, w, mu = _hub(n, hubs, n)
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(bogus_gpu.PrimalFrictionProblem(minv, objA, objB, HA, HB, w, mu))
    rp, cl, vl = oracle.PrimalProblem(minv, objA, objB, HA, HB).assemble()
    x = np.random.default_rng(n).standard_normal(3 * n)
    y = D.multiply(x)
    rp_g, cl_g, vl_g = D.W_lower()
    assert np.array_equal(rp_g, rp) and np.array_equal(cl_g, cl)
    assert np.array_equal(vl_g.reshape(-1), np.asarray(vl).reshape(-1))
    assert np.array_equal(y, oracle.DualProblem(rp, cl, vl, w, mu).spmv(x))


def test_hub_time():
    """3000 contacts of one body, 9 million blocks: 0.22 s with the pattern built on the host; sorting each row's upper half
    in one thread took 2.9 s."""
    import bogus_gpu

    P = bogus_gpu.PrimalFrictionProblem(*_hub(3000, 1, 1))
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(P)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        D.computeFrom(P)
        times.append(time.perf_counter() - t0)
    assert min(times) < 0.2
