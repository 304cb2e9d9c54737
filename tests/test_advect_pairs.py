"""The float-pair forms of the advection passes against the FP64 forms.

tests/kernel_host/advect_fast_harness.cpp runs every pass of
shiokaze_gb300/csrc/advect_fast.cuh on the host beside the FP64 form it
stands for (advect_core.cuh, pinned to the reference by test_kernel_host.py),
from the same state. Every value has to be the same bits, for all inputs;
ordinary flows leave few elements to the FP64 form. The GPU tests run the
same forms against the oracle where they can go wrong: the smallest grid,
ragged edges, velocities from rest to many cells a step.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from shiokaze_gb300 import scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FP = ctypes.POINTER(ctypes.c_float)
U8 = ctypes.POINTER(ctypes.c_ubyte)


@pytest.fixture(scope="module")
def pairs(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("kernel_host") / "libadvect_fast.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-D__host__=",
                           "-D__device__=", "-D__forceinline__=inline", "-I", "/usr/local/cuda/include", "-I",
                           os.path.join(ROOT, "shiokaze_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "kernel_host", "advect_fast_harness.cpp"), "-o", so])
    lib = ctypes.CDLL(so)
    lib.pairs_advect.argtypes = [ctypes.c_int] * 4 + [ctypes.c_double] * 2 + [ctypes.c_int] * 2 + [FP] * 5 + \
        [U8, ctypes.c_float, ctypes.POINTER(ctypes.c_longlong)]
    lib.pairs_division.argtypes = [ctypes.c_double, ctypes.c_longlong, ctypes.POINTER(ctypes.c_double)]
    lib.pairs_division.restype = ctypes.c_longlong
    return lib


def run_pairs(lib, vel, fluid, dx, dt, q, mask=None, bg=0.0, mac=True, trim=1):
    """(values that differ, share of elements left to the FP64 form)"""
    dim = len(vel)
    shape = fluid.shape if dim == 3 else (1,) + fluid.shape[-2:]
    arrs = [np.ascontiguousarray(a, np.float32) for a in (*vel, *([None] * (3 - dim)), fluid, q) if a is not None]
    p = [a.ctypes.data_as(FP) for a in arrs]
    if dim == 2:
        p.insert(2, None)
    m = None if mask is None else np.ascontiguousarray(mask, np.uint8)
    counts = (ctypes.c_longlong * 3)()
    on = lib.pairs_advect(dim, shape[2], shape[1], shape[0], dx, dt, int(mac), trim, *p,
                          None if m is None else m.ctypes.data_as(U8), bg, counts)
    return counts[0], counts[1] / max(1, counts[2]), on


def flow(rng, kind, shape):
    """One velocity component: noise, rest, a few values, uniform, extremes."""
    a = rng.normal(0, 1, shape)
    if kind == "tiny":
        a *= 10.0 ** rng.uniform(-14, -3, shape)
    elif kind == "steps":
        a = rng.choice([0.0, -0.0, 0.25, -0.5, 1.0, 3.0], shape)
    elif kind == "sparse":
        a *= rng.random(shape) < 0.2
    elif kind == "wide":
        a *= 2.0 ** rng.uniform(-140, 60, shape)
    elif kind == "odd":
        a.flat[rng.integers(0, a.size, 5)] = [np.nan, np.inf, -np.inf, 1e38, 1e-45]
    return a.astype(np.float32)


KINDS = ["noise", "tiny", "steps", "sparse", "wide", "odd"]


@pytest.mark.parametrize("seed", range(24))
def test_pairs_equal_fp64(pairs, seed):
    rng = np.random.default_rng(seed)
    dim = 3 if seed % 3 else 2
    n = [int(x) for x in rng.integers(2, 20, 3)]
    nz = n[2] if dim == 3 else 1
    kind = KINDS[seed % 6]
    shapes = [(nz, n[1], n[0] + 1), (nz, n[1] + 1, n[0]), (nz + 1, n[1], n[0])][:dim]
    vel = [flow(rng, kind if rng.random() < 0.7 else "noise", s) for s in shapes]
    dx = [1.0 / 16, 1.0 / 37, float(rng.uniform(0.01, 0.2))][seed % 3 if seed % 2 else (seed // 2) % 3]
    dt = [1.0 / 60, 1.0 / 64, 0.0469, 3.0 / 64][(seed // 4) % 4]
    cells = (nz, n[1], n[0])
    fluid = (-dx * rng.choice([1.0, 1.7, 0.1]) + rng.normal(0, 1, cells) * dx * 10.0 ** rng.uniform(-9, 0)).astype(np.float32)
    q = flow(rng, KINDS[(seed // 5) % 6], cells)
    mask = (rng.random(cells) < 0.8).astype(np.uint8) if seed % 4 == 1 else None
    for mac in (True, False):
        bad, _, on = run_pairs(pairs, vel, fluid, dx, dt, q, mask, 0.5, mac, int(rng.integers(0, 3)))
        assert on and bad == 0


@pytest.mark.parametrize("dx", [1.0 / 48, 1.0 / 64])
def test_pairs_decide_nearly_all(pairs, dx):
    """On a moving field hardly any element needs the FP64 form: by the error
    bounds, 8 roundings of 2^-18 to 2^-20 each, and the displacement's."""
    rng = np.random.default_rng(5)
    n = 40
    sc = scenes.smoke3(n, seed=2, sigma=1.0)
    q = rng.random(sc.fluid.shape, dtype=np.float32)
    bad, left, on = run_pairs(pairs, (sc.u, sc.v, sc.w), sc.fluid, dx, 1.0 / 60, q)
    assert on and bad == 0 and left < 2e-3


def test_division_by_known_divisor(pairs):
    rng = np.random.default_rng(1)
    for dx in [1.0 / 3, 1.0 / 777, 0.1, np.nextafter(1.0, 0), np.nextafter(0.5, 1), 1e-3, *rng.uniform(1e-4, 1, 40)]:
        x = rng.normal(0, 1, 200000) * 2.0 ** rng.uniform(-60, 30, 200000)
        x[:100] = np.arange(100) * dx  # quotients at and beside integers
        assert pairs.pairs_division(float(dx), x.size, x.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dim,n,kind,dx", [(3, (2, 2, 2), "noise", 0.25), (3, (33, 2, 17), "steps", 1.0 / 32),
                                           (3, (31, 20, 9), "tiny", 1.0 / 33), (3, (65, 12, 7), "wide", 1.0 / 64),
                                           (3, (40, 24, 18), "odd", 0.013), (2, (2, 2, 1), "noise", 0.5),
                                           (2, (257, 33, 1), "sparse", 1.0 / 257), (2, (64, 65, 1), "tiny", 1.0 / 64)])
def test_gpu_matches_oracle(dim, n, kind, dx):
    import oracle
    import shiokaze_gb300 as gb
    rng = np.random.default_rng(sum(n))
    nx, ny, nz = n
    shapes = ([(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)] if dim == 3 else [(ny, nx + 1), (ny + 1, nx)])
    cells = (nz, ny, nx) if dim == 3 else (ny, nx)
    vel = [flow(rng, kind, s) for s in shapes]
    fluid = (-dx + rng.normal(0, 1, cells) * dx).astype(np.float32)
    q = rng.normal(0, 1, cells).astype(np.float32)
    mask = (rng.random(cells) < 0.8).astype(np.uint8)
    want = (oracle.advect3 if dim == 3 else oracle.advect2)(*vel, fluid, dx, 1.0 / 60, q=q, q_mask=mask, q_bg=0.25)
    adv = gb.MacAdvection3(nx, ny, nz, dx) if dim == 3 else gb.MacAdvection2(nx, ny, dx)
    got, qo = [a.copy() for a in vel], q.copy()
    adv.advect_step(tuple(got), fluid, 1.0 / 60, scalar=qo, mask=mask, background=0.25)
    for a, b in zip((*got, qo), want):
        b = np.asarray(b).reshape(a.shape)
        assert np.array_equal(np.isnan(a), np.isnan(b))
        keep = ~np.isnan(a)
        assert np.array_equal(a.view(np.uint32)[keep], b.view(np.uint32)[keep])
