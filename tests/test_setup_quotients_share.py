"""How often quot_round (shiokaze_gb300/csrc/gbp_exact.cuh) leaves the quotient to the
FP64 form, on the host: never more than half of the values (where dt / dx is a short
fraction, half of the products can be ties), all of them where dt / dx leaves the
pair's range. Without that bound a form that never decides would pass the comparison
of values."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FP = ctypes.POINTER(ctypes.c_float)


@pytest.fixture(scope="module")
def quot(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("quot") / "libquot.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                           os.path.join(ROOT, "shiokaze_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "kernel_host", "quot_harness.cpp"), "-o", so, "-lm"])
    lib = ctypes.CDLL(so)
    lib.host_quot.argtypes = [ctypes.c_double] * 2 + [FP, FP, ctypes.c_longlong, ctypes.POINTER(ctypes.c_longlong)]
    lib.host_quot.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("dt,dx,least,most", [(0.0173, 1 / 128, 0.0, 0.5), (0.0231, 1 / 96, 0.0, 0.5),
                                              (-0.0117, 0.031, 0.0, 0.5), (0.01, 1 / 75, 0.0, 0.5),
                                              (1e-20, 1.0, 1.0, 1.0), (1.0, 1e-13, 1.0, 1.0)])
def test_share_left_to_fp64(quot, dt, dx, least, most):
    rng = np.random.default_rng(23)
    f = rng.standard_normal(1 << 20).astype(np.float32)
    f[f == 0] = 1.0
    rho = np.where(rng.random(f.size) < 0.5, 1.0, 0.01 + 0.99 * rng.random(f.size)).astype(np.float32)
    left = ctypes.c_longlong(0)
    assert quot.host_quot(dt, dx, f.ctypes.data_as(FP), rho.ctypes.data_as(FP), f.size, ctypes.byref(left)) == 0
    assert least * f.size <= left.value <= most * f.size
