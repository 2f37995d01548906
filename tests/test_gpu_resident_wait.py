"""A wait that runs out in one CTA of a cluster (csrc/resident.cuh): the others
learn of it with the next sum over the group and not before, so that all of them
can leave at the same point, and the sums are unharmed.  The wait is for 16
bytes that nobody sends, with a limit of 64 tries."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory, cuda_lib):
    from coolpdlp import build as B
    so = str(tmp_path_factory.mktemp("wait") / "resident_wait.so")
    subprocess.check_call([B.nvcc(), *B.ARCH, "-std=c++17", "-O1", "-Xcompiler", "-fPIC", "-shared",
                           "--expt-relaxed-constexpr", "-I", B.CSRC, "-I",
                           os.path.join(os.path.dirname(HERE), "include"),
                           os.path.join(HERE, "native", "resident_wait.cu"), "-o", so])
    return ctypes.CDLL(so)


@pytest.mark.parametrize("wait_rank", [-1, 0, 1])
def test_a_group_learns_of_a_wait_that_ran_out(lib, wait_rank):
    out = np.full((2, 2, 4), np.nan)
    assert lib.resident_wait(wait_rank, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    for rank in range(2):
        before, after, first, last = out[rank, 0]
        assert before == (1.0 if rank == wait_rank else 0.0)
        assert after == (0.0 if wait_rank < 0 else 1.0)
        assert (first, last) == (512.0, 2560.0)
        # and it is not forgotten; a second wait returns at once
        before, after, first, last = out[rank, 1]
        assert before == after == (0.0 if wait_rank < 0 else 1.0)
        assert (first, last) == (512.0, 2560.0)
