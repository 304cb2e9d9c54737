"""The coarse-level kernels' grid barrier over the wrap of its 32-bit count, which a
long solve reaches: blocks pass when all have arrived and not before."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("barrier") / "libbarrier.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I",
                           os.path.join(ROOT, "shiokaze_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "kernel_host", "barrier_harness.cpp"), "-o", so])
    lib = ctypes.CDLL(so)
    lib.host_barriers.argtypes = [ctypes.c_uint, ctypes.c_uint, ctypes.c_int, ctypes.c_void_p]
    lib.host_barriers.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("grid", [1, 2, 3, 64, 65, 152, 304, 456])
def test_barrier_over_the_wrap(lib, grid):
    rng = np.random.default_rng(grid)
    span = 1 << (grid - 1).bit_length()
    for start in (0, 2**32 - span, 2**32 - 2 * span):
        order = np.stack([rng.permutation(grid) for _ in range(4)]).astype(np.int32)
        assert lib.host_barriers(start, grid, 4, order.ctypes.data) == 0
