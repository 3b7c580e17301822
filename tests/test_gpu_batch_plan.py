"""The plan of a batched solve is a small part of setting the batch."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _best(call, times=7):
    out = []
    for _ in range(times):
        t0 = time.perf_counter()
        call()
        out.append(time.perf_counter() - t0)
    return min(out)


def test_plan_of_many_problems():
    """20 000 problems of 20 contacts against the same matrix as one problem, which is too large to plan: what is left of
    setting the batch (reading W's structure, checking it, the uploads) is the same. 1.3 times as long measured; 6.6 with
    the CTAs sorted anew for every problem and candidate."""
    import bogus_gpu

    problems, n = 20000, 20
    D = bogus_gpu.DualFrictionProblem()
    rp = np.concatenate([[0], np.cumsum(np.arange(problems * n) % n + 1)]).astype(np.int32)  # dense lower triangles
    cl = np.concatenate([np.arange(i // n * n, i + 1) for i in range(n)]).astype(np.int32)
    cl = (cl[None, :] + n * np.arange(problems)[:, None]).reshape(-1).astype(np.int32)
    vl = np.tile(0.01 * np.eye(3), (len(cl), 1, 1))
    vl[rp[1:] - 1] = np.eye(3)
    D.set(rp, cl, vl, np.ones(3 * problems * n), np.full(problems * n, 0.5))
    many = np.arange(0, problems * n + 1, n, dtype=np.int32)
    one = np.array([0, problems * n], np.int32)
    D.setBatch(many)
    t_one = _best(lambda: D.setBatch(one))
    t_many = _best(lambda: D.setBatch(many))
    assert t_many < 2.5 * t_one, (t_many, t_one)
