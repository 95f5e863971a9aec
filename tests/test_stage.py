"""Staging of pageable rows on the host: with as many threads as there is memory
for, every byte arrives and no thread is left behind."""
import ctypes
import os
import subprocess
import sys

import pytest

from supergwas_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(HERE, "native", "_build", "libstage_check.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic-functions", "-I" + cuda, "-o", out,
                    os.path.join(HERE, "native", "stage_check.cpp"), "-lpthread"], check=True)
    return out


# the block flags and the thread list take the first two allocations, every thread one more
@pytest.mark.parametrize("allocations", [-1, 0, 1, 2, 3, 5])
@pytest.mark.parametrize("size", [1, (4 << 20) + 1, (37 << 20) + 5])
def test_every_byte_arrives(lib, size, allocations):
    """In a process of its own: a joinable thread that is destroyed ends it."""
    code = (f"import ctypes, os; f = ctypes.CDLL({lib!r}, mode=os.RTLD_LAZY).stage_call; "
            f"f.argtypes = [ctypes.c_uint64, ctypes.c_int]; print(f({size}, {allocations}))")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == "0"
