"""Device code that orders the warps of a CTA, run on the host with a thread per lane (tests/hostwarp): what it does not
order, slow lanes of the simulation bring into the wrong order."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "hostwarp", "hostwarp.cpp")
CSRC = os.path.join(HERE, "..", "so-bogus_gb300", "csrc")


@pytest.fixture(scope="module")
def hostwarp(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hostwarp") / "libhostwarp.so")
    subprocess.run(["g++", "-O1", "-std=c++20", "-fPIC", "-shared", "-pthread", "-I" + CSRC, "-o", out, SRC], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("chunks", [1, 2, 9, 16])
def test_cluster_side_work_precedes_the_decision(hostwarp, chunks):
    """The side work of a reduction (the momentum weight, the step that a rejection takes) is done before the decision
    that reads it, and reads the previous decision's values."""
    assert hostwarp.hw_cluster_reduce(chunks, 8) == 0


@pytest.mark.parametrize("late", [0, 1, 1 << 5, 1 << 31, 0xffffffff])
@pytest.mark.parametrize("stopped", [0, 1 << 9])
@pytest.mark.parametrize("before", [0, 7])
def test_a_warp_that_gives_up_says_why(hostwarp, late, stopped, before):
    """Whichever lane's wait runs out, the whole warp leaves and the status word says so (an earlier reason stays)."""
    status = ctypes.c_int(before)
    gave = hostwarp.hw_warp_gives_up(ctypes.c_uint(late), ctypes.c_uint(stopped), ctypes.byref(status))
    assert gave == (1 if late or stopped else 0)
    assert status.value == (before or (5 if late else 0))


@pytest.mark.parametrize("at", [[], [0], [1], [17, 40], [0, 32], [33], list(range(64))])
def test_every_cta_of_a_cluster_sees_the_same_maximum(hostwarp, at):
    """A maximum over values with NaN among them depends on the lane that holds it; the CTAs of a cluster have to take one
    lane's, the first as the other kernels do, or their decisions part."""
    values = np.linspace(1.0, 2.0, 64)
    values[at] = np.nan
    totals = np.full(2, 7.0)
    hostwarp.hw_cluster_max(values.ctypes.data_as(ctypes.c_void_p), totals.ctypes.data_as(ctypes.c_void_p))
    assert np.array_equal(totals[:1], totals[1:], equal_nan=True)

    def butterfly(v):
        for off in (16, 8, 4, 2, 1):
            o = v[np.arange(32) ^ off]
            v = np.where(v < o, o, v)
        return v[0]

    # two chunks, a stripe each: 0, then the chunk's maximum where it is not below; the stripes left to right
    total = None
    for s in range(8):
        v = butterfly(values[32 * s:32 * s + 32]) if s < 2 else 0.0
        v = 0.0 if v < 0.0 else v
        total = v if total is None else total if v < total else v
    assert np.array_equal(totals[0], total, equal_nan=True)
