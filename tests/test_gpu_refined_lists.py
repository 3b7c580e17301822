"""A refined solve whose parts run on grids of different sizes keeps the chunk lists of each between calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uploads(torch, n):
    """Host-to-device copies of a repeated refined solve of n contacts."""
    import bogus_gpu
    from bogus_gpu import generator

    D = bogus_gpu.DualFrictionProblem()
    D.computeFrom(bogus_gpu.PrimalFrictionProblem.from_generated(generator.grid(n // 4, n, seed=1)))
    pg = bogus_gpu.ProjectedGradient()
    pg.setTol(1e-14)
    pg.setMaxIters(3)
    pg.setMixedPrecision(True, 4)
    pg.setFp32CorrectionProducts(2)
    r = np.zeros(3 * n)
    for _ in range(2):
        D.solveWith(pg, r.copy(), staticProblem=True)
    kinds = [torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]
    for _ in range(2):  # a process's first recording may miss the device's side
        with torch.profiler.profile(activities=kinds) as prof:
            D.solveWith(pg, r.copy(), staticProblem=True)
            torch.cuda.synchronize()
    return sum(e.count for e in prof.key_averages() if "HtoD" in e.key)


def test_lists_are_kept():
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda:0")
    shared = _uploads(torch, 20000)  # both parts on one CTA per SM: the lists were built once
    if shared == 0:
        pytest.skip("no copies recorded")
    assert _uploads(torch, 45000) == shared  # the FP64 check on two CTAs per SM
