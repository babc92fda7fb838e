"""The count by which the CTA of a block's last chunk knows itself (block means of N^-1), over
more than 2^32 arrivals: an operator that a serving process keeps gets there within the hour."""
import ctypes as ct
import os
import subprocess

import pytest

from midapack_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_last_arrival_past_the_counts_range(gpu_ctx, tmp_path):
    so = str(tmp_path / "libarrival_count.so")
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-cudart", "shared", "-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC,
                    os.path.join(HERE, "arrival_count.cu"), "-o", so], check=True)
    f = ct.CDLL(so).arrival_count
    f.argtypes = [ct.c_uint32, ct.c_longlong, ct.POINTER(ct.c_ulonglong), ct.POINTER(ct.c_int)]
    n = 147                                   # not a power of two
    rounds = (1 << 32) // n + 2
    lasts, which = ct.c_ulonglong(), (ct.c_int * n)()
    assert f(n, rounds, ct.byref(lasts), which) == 0
    assert lasts.value == rounds
    assert list(which) == [0] * (n - 1) + [1]
