"""The setup's quotients without FP64 divisions: quot_round and div_round of
shiokaze_gb300/csrc/gbp_exact.cuh on the host against the FP64 expressions they
stand for, bit for bit; and, on the GPU, the face-first setup and velocity
update against the allocation-free entry point, which evaluates every face by
those expressions, and against the oracle's assembly on noise that cuts most
faces of a million (the queue of cut faces fills and empties), on cell sizes
that are and are not powers of two."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from shiokaze_gb300 import scenes

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
    lib.host_div.argtypes = [ctypes.c_double, FP, ctypes.c_longlong]
    lib.host_quot.restype = lib.host_div.restype = ctypes.c_longlong
    return lib


def _floats(rng, n):
    f = rng.standard_normal(n).astype(np.float32) * np.exp2(rng.integers(-30, 31, n)).astype(np.float32)
    f[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, 3.4e38, 1.0]
    f[8: n // 8] = rng.integers(-4096, 4097, n // 8 - 8)  # short significands: ties and exact quotients
    return f


@pytest.mark.parametrize("dt,dx", [(0.01, 1 / 128), (0.01, 1 / 75), (1 / 30, 1 / 147), (0.0375, 1 / 3), (0.25, 1 / 96),
                                   (1e-3, 0.1), (-0.01, 1 / 61), (1e-20, 1.0)])
def test_quotients_equal_fp64(quot, dt, dx):
    rng = np.random.default_rng(17)
    f = _floats(rng, 1 << 20)
    rho = np.where(rng.random(f.size) < 0.5, 1.0, rng.random(f.size) + 1e-6).astype(np.float32)
    rho = np.minimum(rho, np.float32(1.0))
    left = ctypes.c_longlong(0)  # many where dt/dx is nearly a short fraction (0.01 * 75): ties
    assert quot.host_quot(dt, dx, f.ctypes.data_as(FP), rho.ctypes.data_as(FP), f.size, ctypes.byref(left)) == 0
    x = f[np.isfinite(f)].copy()
    assert quot.host_div(dx, x.ctypes.data_as(FP), x.size) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n,dx", [((33, 17, 40), 1 / 40), ((33, 17, 40), 1 / 32), ((1, 5, 9), 1 / 9), ((40, 20, 40), 1 / 75)])
@pytest.mark.parametrize("cut", [0.0, 1.0])
def test_faces_equal_single_pass(n, dx, cut):
    import torch

    import shiokaze_gb300 as gb
    sc = scenes.liquid3(n, seed=3)
    rng = np.random.default_rng(5)
    noise = lambda a: a + cut * dx * rng.standard_normal(a.shape).astype(np.float32)  # noqa: E731
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    solid, fluid = dev(noise(sc.solid)), dev(noise(sc.fluid))
    a, b = ([dev(x) for x in (sc.u, sc.v, sc.w)] for _ in range(2))
    pa, pb = (torch.empty(sc.fluid.shape, device="cuda") for _ in range(2))
    opts = dict(Residual=1e-6, MaxIterations=30)
    pj = gb.MacProject3(*n, dx, **opts)
    ra = pj.project(sc.dt, a, solid, fluid, pressure_out=pa)
    lib = gb.load_library()
    st, prm = gb.Stats(), gb.make_params(**opts)
    vp = ctypes.c_void_p
    lib.gbp_project_device_static.argtypes = [ctypes.c_int] * 4 + [ctypes.c_double] * 2 + [vp] * 5 + \
        [ctypes.POINTER(gb.Params), vp, ctypes.POINTER(gb.Stats), vp]
    torch.cuda.synchronize()
    rb = lib.gbp_project_device_static(3, *n, dx, sc.dt, solid.data_ptr(), fluid.data_ptr(), *(t.data_ptr() for t in b),
                                       ctypes.byref(prm), pb.data_ptr(), ctypes.byref(st),
                                       vp(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert ra == rb and pj.stats.iterations == st.iterations
    for x, y in zip([pa, *a], [pb, *b]):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))
    pj.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dx", [1 / 128, 1 / 101])
def test_queue_of_cut_faces(dx):
    import oracle
    import shiokaze_gb300 as gb
    n = (101, 100, 128)
    sc = scenes.liquid3(n, seed=3)
    rng = np.random.default_rng(6)
    noise = lambda a: (a + dx * rng.standard_normal(a.shape)).astype(np.float32)  # noqa: E731
    solid, fluid = noise(sc.solid), noise(sc.fluid)
    pj = gb.MacProject3(*n, dx)
    got = pj.debug_assemble(sc.dt, (sc.u, sc.v, sc.w), solid, fluid)
    pj.close()
    port = oracle.PortProjector(3, *n, dx)
    want = port.assemble(sc.dt, solid, fluid, sc.u, sc.v, sc.w)
    port.close()
    for k in ("diag", "cpx", "cpy", "cpz", "b"):
        assert np.array_equal(got[k], want[k]), k
