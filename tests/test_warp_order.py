"""Device code that orders the warps of a CTA, run on the host with a thread per lane (tests/hostwarp): what it does not
order, slow lanes of the simulation bring into the wrong order."""
import ctypes
import os
import subprocess

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
