"""The compliance term with and without a host copy of W's lower triangle: the same triangle, the same solves, and no
download where there is none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nbodies", [(1, 2), (31, 12), (128, 50), (129, 300), (500, 200)])
@pytest.mark.parametrize("assembled", [True, False])
def test_same_triangle(n, nbodies, assembled):
    import bogus_gpu
    from bogus_gpu import generator

    d = generator.random_pairs(nbodies, n, seed=n)
    c = np.random.default_rng(n).uniform(0.0, 0.1, n)
    P = bogus_gpu.PrimalFrictionProblem.from_generated(d)
    out = []
    for host_first in (False, True):
        D = bogus_gpu.DualFrictionProblem()
        D.computeFrom(P)
        if not assembled:
            D.set(*D.W_lower(), d.b, d.mu)
        if host_first:
            before = D.W_lower()
        for _ in range(2):
            D.add_compliance(c)
        low = D.W_lower()
        gs = bogus_gpu.GaussSeidel()
        gs.setMaxIters(10)
        r = np.zeros(3 * n)
        out.append((low, D.solveWith(gs, r), r))
    assert all(np.array_equal(a, b) for a, b in zip(out[0][0], out[1][0]))
    assert out[0][1] == out[1][1] and np.array_equal(out[0][2], out[1][2])
    expected = before[2].copy()
    k = before[0][1:] - 1  # the diagonal blocks end the rows
    for e in range(3):
        expected[k, e, e] = (expected[k, e, e] + c) + c
    assert np.array_equal(out[1][0][2], expected)


def test_no_download():
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda:0")
    import bogus_gpu
    from bogus_gpu import generator

    P = bogus_gpu.PrimalFrictionProblem.from_generated(generator.random_pairs(200, 500, seed=1))
    D = bogus_gpu.DualFrictionProblem()
    kinds = [torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]
    for _ in range(2):  # a process's first recording may miss the device's side
        D.computeFrom(P)
        with torch.profiler.profile(activities=kinds) as prof:
            D.add_compliance(0.05)
            torch.cuda.synchronize()
    down = sum(e.count for e in prof.key_averages() if "DtoH" in e.key)
    if down == 0:
        pytest.skip("no copies recorded")
    assert down == 1  # the places of the diagonal blocks
