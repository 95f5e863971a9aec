"""A refinement candidate of a many-phenotype launch holds its k-mer in 47 bits
(bit 47 marks an open gate): calls of more k-mers are refused."""
import ctypes
import os
import subprocess

from supergwas_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
ERR_CUDA, ERR_UNSUPPORTED = 2, 6  # include/kgwas_cuda.h


def test_number_of_kmers():
    out = os.path.join(HERE, "native", "_build", "libmulti_limits_check.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic-functions", "-I" + cuda, "-o", out,
                    os.path.join(HERE, "native", "multi_limits_check.cpp"), "-lpthread"], check=True)
    call = ctypes.CDLL(out, mode=os.RTLD_LAZY).multi_call
    call.argtypes = [ctypes.c_uint64]
    assert call((1 << 47) - 1) == ERR_CUDA  # past the checks
    assert call(1 << 47) == call(1 << 60) == ERR_UNSUPPORTED
