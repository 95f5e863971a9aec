"""A pair kernel that does not launch makes the call fail (kg_pairs_run_host on
the host, with stand-ins for the CUDA calls)."""
import ctypes
import os
import subprocess

import pytest

from supergwas_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
OK, ERR_CUDA = 0, 2  # include/kgwas_cuda.h
INVALID_VALUE, OUT_OF_MEMORY = 1, 2  # cudaError_t


@pytest.fixture(scope="module")
def pairs_call():
    out = os.path.join(HERE, "native", "_build", "libpairs_launch_check.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic-functions", "-I" + cuda, "-o", out,
                    os.path.join(HERE, "native", "pairs_launch_check.cpp"), "-lpthread"], check=True)
    fn = ctypes.CDLL(out).pairs_call

    def call(*args):
        ran = (ctypes.c_int * 2)()
        return fn(*args, ran), list(ran)
    return call


@pytest.mark.parametrize("fs", [0, 1])
def test_launch_results(pairs_call, fs):
    assert pairs_call(fs, 0, 0) == (OK, [fs, 1])
    for code in (INVALID_VALUE, OUT_OF_MEMORY):
        rc, ran = pairs_call(fs, code, 0)
        assert rc == ERR_CUDA and ran == [fs, 0]
    assert pairs_call(fs, 0, INVALID_VALUE)[0] == ERR_CUDA
