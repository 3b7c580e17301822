"""The Delassus assembly whose pattern is built on the device, against the oracle's, bit for bit: dof counts other than
the specialised 6, contacts of a body with itself and with the ground, bodies without contacts, a body in every contact
(rows that meet all others), and a single contact; twice on one handle, so that a smaller problem follows a larger."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _primal(n, nbodies, ndof, seed, hub):
    rng = np.random.default_rng(seed)
    objA = rng.integers(0, nbodies, n).astype(np.int32)
    objB = rng.integers(-1, nbodies, n).astype(np.int32)
    if hub:
        objA[:] = nbodies - 1
    objB[:: 7] = objA[:: 7]  # a body with itself: its block counts once
    HA, HB = rng.standard_normal((2, n, 3, ndof))
    HB[objB < 0] = 0.0
    R = rng.standard_normal((nbodies, ndof, ndof))
    minv = np.einsum("bij,bkj->bik", R, R) + np.eye(ndof)
    return minv, objA, objB, HA, HB, rng.standard_normal(3 * n), rng.uniform(0.3, 0.8, n), rng.standard_normal(nbodies * ndof)


@pytest.mark.parametrize("ndof", [1, 3, 6, 12])
def test_assembly(oracle, ndof):
    import bogus_gpu

    D = bogus_gpu.DualFrictionProblem()
    for n, nbodies, hub in ((300, 90, False), (129, 500, False), (70, 5, True), (1, 2, False)):
        minv, objA, objB, HA, HB, w, mu, f = _primal(n, nbodies, ndof, 10 * n + ndof, hub)
        D.computeFrom(bogus_gpu.PrimalFrictionProblem(minv, objA, objB, HA, HB, w, mu, f=f))
        rp, cl, vl = oracle.PrimalProblem(minv, objA, objB, HA, HB).assemble()
        rp_g, cl_g, vl_g = D.W_lower()
        assert np.array_equal(rp_g, rp) and np.array_equal(cl_g, cl)
        assert np.array_equal(vl_g.reshape(-1), np.asarray(vl).reshape(-1))
        x = np.random.default_rng(n).standard_normal(3 * n)
        assert np.array_equal(D.multiply(x), oracle.DualProblem(rp, cl, vl, w, mu).spmv(x))
