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


@pytest.mark.parametrize("n,nbodies", [(31, 12), (33, 11), (255, 90), (256, 300), (257, 90), (481, 160), (512, 200), (513, 200)])
def test_cluster(oracle, n, nbodies):
    """Problems of one cluster: one CTA, one and two chunks per stripe of the sums, the last size and the first past it."""
    D, O = _pair(oracle, n, nbodies, 70 + n)
    for variant, coulomb, inf_norm in ((3, False, True), (3, True, False), (4, False, False), (4, True, True), (1, False, False)):
        _compare(D, O, n, variant, coulomb, inf_norm, 60, np.zeros(3 * n))


@pytest.mark.parametrize("n", [16 * 32 * SM, 16 * 32 * SM + 1])
def test_general(oracle, n):
    """The general kernel on both sides of the line between its two register budgets (kernels_pg.cu)."""
    D, O = _pair(oracle, n, n // 4, 11)
    for variant, coulomb in ((3, False), (4, True), (1, False)):
        _compare(D, O, n, variant, coulomb, False, 6, np.zeros(3 * n))


@pytest.mark.parametrize("sizes", [[1, 31, 32, 33, 160, 161, 1], [16] * 40 + [700, 340, 5, 64], [0, 50, 0, 200]])
def test_batch(oracle, sizes):
    """Batches whose problems span one and several CTAs, several problems per CTA, and empty problems: each problem as the
    oracle solves it alone."""
    import bogus_gpu
    from bogus_gpu import generator

    parts = [generator.random_pairs(max(2, n // 3), n, seed=90 + k) if n else None for k, n in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum([d.nbodies if d else 0 for d in parts])])
    live = [(d, o) for d, o in zip(parts, off) if d]
    cat = lambda f: np.concatenate([f(d, o) for d, o in live])  # noqa: E731
    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(bogus_gpu.PrimalFrictionProblem(
        cat(lambda d, o: d.minv), cat(lambda d, o: d.objA + o), cat(lambda d, o: np.where(d.objB >= 0, d.objB + o, -1)),
        cat(lambda d, o: d.HA), cat(lambda d, o: d.HB), cat(lambda d, o: d.b), cat(lambda d, o: d.mu)))
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    D.setBatch(ptr)
    for variant, static in ((3, True), (4, False), (1, True)):
        pg = bogus_gpu.ProjectedGradient()
        pg.setDefaultVariant(variant)
        pg.setMaxIters(60)
        pg.setTol(1e-8)
        r = np.zeros(3 * ptr[-1])
        res, its = D.solveBatchWith(pg, r, staticProblem=static)
        for p, d in enumerate(parts):
            if d is None:
                continue
            rp, cl, vl = oracle.PrimalProblem(d.minv, d.objA, d.objB, d.HA, d.HB).assemble()
            ro, xo, io = oracle.DualProblem(rp, cl, vl, d.b, d.mu).solve_pg(
                np.zeros(3 * d.n), variant=variant, coulomb=not static, tol=1e-8, max_iters=60)
            assert res[p] == ro and its[p] == io and np.array_equal(r[3 * ptr[p]:3 * ptr[p + 1]], xo), (p, variant)


@pytest.mark.parametrize("n,nbodies", [(1, 2), (33, 30), (161, 120)])
def test_adjoint(oracle, n, nbodies):
    """The adjoint's resident kernel (a partial chunk, one past a chunk, several CTAs) against the dense gradients, within
    the adjoint tests' 1e-8 of the largest entry (conjugate gradients stop at 1e-13)."""
    import adjoint
    import bogus_gpu

    D, _ = _pair(oracle, n, nbodies, 60 + n)
    D.add_compliance(0.05)
    rp, cl, vl = D.W_lower()
    b, mu = np.empty(3 * n), np.empty(n)
    assert bogus_gpu.lib().bogus_gpu_get_dual_rhs(D.handle, b.ctypes.data, mu.ctypes.data) == 0
    _, r, _ = oracle.DualProblem(rp, cl, vl.reshape(-1), b, mu).solve_gs(np.zeros(3 * n), coulomb=False, tol=1e-32,
                                                                         max_iters=3000, coloring=False)
    W = np.zeros((3 * n, 3 * n))
    for i in range(n):
        for k in range(rp[i], rp[i + 1]):
            j = cl[k]
            W[3 * i:3 * i + 3, 3 * j:3 * j + 3] = vl[k]
            W[3 * j:3 * j + 3, 3 * i:3 * i + 3] = vl[k].T
    g = np.random.default_rng(n).standard_normal(3 * n)
    s_o, dmu_o, _ = adjoint.implicit_gradient(W, b, mu, r, g)
    s, dmu = D.adjoint(r, g, tol=1e-13)
    assert np.abs(s - s_o).max() <= 1e-8 * max(np.abs(s_o).max(), 1e-300)
    assert np.abs(dmu - dmu_o).max() <= 1e-8 * max(1.0, np.abs(dmu_o).max())


@pytest.mark.parametrize("n,nbodies", [(1, 2), (33, 30), (70, 4), (64, 24), (32 * SM + 1, 1600), (8 * 32 * SM + 1, 13000),
                                       (49999, 16000), (52000, 10000)])
def test_refined(oracle, n, nbodies):
    """The FP32-refined solve (kernels_pg_resident32.cu; the last two sizes around the shared-memory limit): FP32 part,
    iterations with FP32 correction products and the FP64 check as the oracle's restatements of the three, one after the
    other."""
    import bogus_gpu

    D, O = _pair(oracle, n, nbodies, 50 + n)
    first, budget, refresh = (60, 40, 7) if n < 1000 else (12, 10, 4)
    for static in (True, False):
        pg = bogus_gpu.ProjectedGradient()
        pg.setTol(1e-12)
        pg.setMaxIters(first)
        pg.setMixedPrecision(True, budget)
        pg.setFp32CorrectionProducts(refresh)
        r = np.zeros(3 * n)
        res = D.solveWith(pg, r, staticProblem=static)
        st = D.solve_stats()
        _, x, k = O.solve_pg_fp32(np.zeros(3 * n), coulomb=not static, tol=1e-12, max_iters=first, stall_iters=4)
        assert k == st["iterations"] - st["refine_iterations"]
        _, x, ith = O.solve_pg(x, variant=3, coulomb=not static, tol=1e-12, max_iters=budget, hy_refresh=refresh)
        assert ith == st["fp32_product_iterations"]
        res_o, x, it = O.solve_pg(x, variant=3, coulomb=not static, tol=1e-12, max_iters=max(1, budget - ith))
        assert it == st["refine_iterations"] - ith and res == res_o and np.array_equal(r, x)


@pytest.mark.parametrize("variant", [1, 4])  # Descent, SPG
def test_refined_variants(oracle, variant):
    """The FP32 part of the other variants against the same solve as a batch of one (k_pg_batch, the plain arrays)."""
    import bogus_gpu

    n = 777
    D, _ = _pair(oracle, n, 300, 3)
    pg = bogus_gpu.ProjectedGradient()
    pg.setDefaultVariant(variant)
    pg.setTol(1e-11)
    pg.setMaxIters(80)
    pg.setMixedPrecision(True, 20)
    a, b = np.zeros(3 * n), np.zeros(3 * n)
    res = D.solveWith(pg, a, staticProblem=True)
    its = D.last_iterations
    D.setBatch(np.array([0, n], dtype=np.int32))
    rb, ib = D.solveBatchWith(pg, b, staticProblem=True)
    assert rb[0] == res and ib[0] == its and np.array_equal(a, b)
