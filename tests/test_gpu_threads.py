"""Handles are independent: host threads that solve problems of different sizes at the same time, each on a handle of its
own, get what each gets alone. The sizes reach the kernels whose shared memory depends on the problem with their largest
and smallest launches."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SM = 152  # GB300


def _dual(n, nbodies, seed):
    import bogus_gpu
    from bogus_gpu import generator

    d = (generator.random_pairs if n < 1000 else generator.grid)(nbodies, n, seed=seed)
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(bogus_gpu.PrimalFrictionProblem.from_generated(d))
    return D


def _pg_call(n, nbodies, mixed=False):
    import bogus_gpu

    D = _dual(n, nbodies, n)
    pg = bogus_gpu.ProjectedGradient()
    pg.setTol(1e-14)
    pg.setMaxIters(3)
    if mixed:
        pg.setMixedPrecision(True, 3)
        pg.setFp32CorrectionProducts(2)

    def call():
        r = np.zeros(3 * n)
        return D.solveWith(pg, r, staticProblem=True), r

    return call


def _batch_call(sizes):
    import bogus_gpu
    from bogus_gpu import generator

    parts = [generator.random_pairs(max(2, n // 3), n, seed=n) for n in sizes]
    off = np.concatenate([[0], np.cumsum([d.nbodies for d in parts])])
    cat = lambda f: np.concatenate([f(d, o) for d, o in zip(parts, off)])  # noqa: E731
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(bogus_gpu.PrimalFrictionProblem(
        cat(lambda d, o: d.minv), cat(lambda d, o: d.objA + o), cat(lambda d, o: np.where(d.objB >= 0, d.objB + o, -1)),
        cat(lambda d, o: d.HA), cat(lambda d, o: d.HB), cat(lambda d, o: d.b), cat(lambda d, o: d.mu)))
    D.setBatch(np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32))
    pg = bogus_gpu.ProjectedGradient()
    pg.setTol(1e-14)
    pg.setMaxIters(3)

    def call():
        r = np.zeros(3 * sum(sizes))
        res, _ = D.solveBatchWith(pg, r, staticProblem=True)
        return res.tolist(), r

    return call


def _adjoint_call(n, nbodies):
    D = _dual(n, nbodies, n)
    D.add_compliance(0.05)
    rng = np.random.default_rng(n)
    r, g = np.abs(rng.standard_normal(3 * n)), rng.standard_normal(3 * n)

    def call():
        db, dmu = D.adjoint(r, g, tol=1e-13, max_iters=3)
        return dmu.tolist(), db

    return call


KINDS = {
    "grid": lambda big: _pg_call(5 * 32 * SM, 8000) if big else _pg_call(520, 700),
    "cluster": lambda big: _pg_call(512, 60) if big else _pg_call(1, 2),
    "refined": lambda big: _pg_call(40000, 10000, True) if big else _pg_call(40, 60, True),
    "batch": lambda big: _batch_call([700, 340, 160, 64] * 8) if big else _batch_call([16, 5, 3]),
    "adjoint": lambda big: _adjoint_call(10000, 3300) if big else _adjoint_call(33, 30),
}


@pytest.mark.parametrize("kind", list(KINDS))
def test_large_and_small_problems_side_by_side(kind):
    calls = [KINDS[kind](True), KINDS[kind](False)]
    alone = [c() for c in calls]
    errors = []

    def worker(call, want, times):
        try:
            for _ in range(times):
                got = call()
                assert got[0] == want[0] and np.array_equal(got[1], want[1])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=worker, args=(c, w, t)) for c, w, t in zip(calls, alone, (300, 600))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
