"""Wait limits of batched solves whose CTAs work through lists of problems: waiting for another CTA's earlier problems is
no hang, however long those take; a wait that nothing feeds ends."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 0.05


@pytest.fixture()
def short_limit():
    import bogus_gpu

    L = bogus_gpu.lib()
    assert L.bogus_gpu_set_wait_limit(0, LIMIT) == bogus_gpu.OK
    yield L
    assert L.bogus_gpu_set_wait_limit(0, 4.0) == bogus_gpu.OK


def _ragged(problems, largest, seed):
    """Problems of 16 to `largest` contacts; every other one separates everywhere and ends in its first iteration."""
    import bogus_gpu
    from bogus_gpu import generator

    rng = np.random.default_rng(seed)
    sizes = np.exp(rng.uniform(np.log(16), np.log(largest + 1), problems)).astype(int)
    parts = [generator.random_pairs(max(2, n // 3), int(n), seed=seed * 1000 + p) for p, n in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum([d.nbodies for d in parts])])
    cat = lambda f: np.concatenate([f(d, o) for d, o in zip(parts, off)])  # noqa: E731
    b = [d.b.reshape(-1, 3).copy() for d in parts]
    for p in range(0, problems, 2):
        b[p] = np.tile([50.0, 0.0, 0.0], (sizes[p], 1))
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(bogus_gpu.PrimalFrictionProblem(
        cat(lambda d, o: d.minv), cat(lambda d, o: d.objA + o), cat(lambda d, o: np.where(d.objB >= 0, d.objB + o, -1)),
        cat(lambda d, o: d.HA), cat(lambda d, o: d.HB), np.concatenate(b).reshape(-1), cat(lambda d, o: d.mu)))
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    D.setBatch(ptr)
    return D, ptr


def test_long_problems_ahead_of_a_shared_one(short_limit):
    import bogus_gpu

    D, ptr = _ragged(256, 1024, 3)
    pg = bogus_gpu.ProjectedGradient()
    pg.setTol(1e-300)  # the separating problems reach 0, the others never this
    pg.setMaxIters(8000)
    r = np.zeros(3 * ptr[-1])
    t0 = time.perf_counter()
    res, its = D.solveBatchWith(pg, r, staticProblem=True)
    assert time.perf_counter() - t0 > 2 * LIMIT  # long enough for the limit to matter
    assert (its[::2] == 0).all() and its[1::2].max() == 8000
    D.setBatchShape(0, 1, 1)  # one CTA per problem: no waits
    r1 = np.zeros(3 * ptr[-1])
    res1, its1 = D.solveBatchWith(pg, r1, staticProblem=True)
    D.setBatchShape(None)
    assert np.array_equal(res, res1) and np.array_equal(its, its1) and np.array_equal(r, r1)


def test_a_wait_that_nothing_feeds_ends(short_limit):
    import bogus_gpu

    D, ptr = _ragged(256, 1024, 4)
    pg = bogus_gpu.ProjectedGradient()
    pg.setTol(1e-8)
    pg.setMaxIters(50)
    good = np.zeros(3 * ptr[-1])
    ref = D.solveBatchWith(pg, good, staticProblem=True)
    r = np.full(3 * ptr[-1], 0.25)
    try:
        assert short_limit.bogus_gpu_test_wait_timeout(D.handle, 1) == bogus_gpu.OK
        t0 = time.perf_counter()
        with pytest.raises(bogus_gpu.BogusGpuError) as e:
            D.solveBatchWith(pg, r, staticProblem=True)
        assert e.value.status == bogus_gpu.TIMEOUT
        assert time.perf_counter() - t0 < 2.0
        assert (r == 0.25).all()
    finally:
        short_limit.bogus_gpu_test_wait_timeout(D.handle, 0)
    again = np.zeros(3 * ptr[-1])
    out = D.solveBatchWith(pg, again, staticProblem=True)
    assert np.array_equal(out[0], ref[0]) and np.array_equal(out[1], ref[1]) and np.array_equal(again, good)
