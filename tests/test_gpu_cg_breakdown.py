"""Plain CG that breaks down: a residual of NaN is GBP_ERR_NAN in every form of
the solve (one launch in a cluster or over the whole GPU, launched iterations),
never a converged one, although |r|_inf passes over NaN."""
import ctypes

import numpy as np
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


# one cluster, every SM, and more rows than the SMs' shared memory holds
@pytest.mark.parametrize("n", [2, 40000, 1000000])
def test_indefinite_rows(n):
    # s.z = 0 in the first iteration: alpha is infinite, then r is NaN
    data = np.ones(n)
    data[1::2] = -1.0
    _, rc, st = gb.csr_cg(np.arange(n + 1), np.arange(n), data, np.ones(n))
    assert rc == gb.GBP_ERR_NAN and not st["converged"]


@pytest.mark.parametrize("n", [2, 40000, 1000000])
@pytest.mark.parametrize("first", [np.nan, 0.0])
def test_nan_right_hand_side(n, first):
    b = np.full(n, np.nan)
    b[0] = first
    _, rc, st = gb.csr_cg(np.arange(n + 1), np.arange(n), np.ones(n), b)
    assert rc == gb.GBP_ERR_NAN and not st["converged"]


@pytest.mark.parametrize("n", [(20, 20, 20), (40, 37, 20)])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_grid(n, value):
    import torch
    sc = scenes.smoke3(n, seed=2)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    solid, fluid, p = dev(sc.solid), dev(sc.fluid), torch.empty(sc.fluid.shape, device="cuda")
    vel = [dev(a) for a in (sc.u, sc.v, sc.w)]
    if np.isnan(value):
        vel[0].fill_(value)  # every row's right-hand side
    else:
        vel[0][3, 4, 5] = value  # two rows', away from the solid
    pj = gb.projector_for(sc, Residual=1e-6)
    other = [a.clone() for a in vel]
    assert pj.project(sc.dt, vel, solid, fluid, pressure_out=p) == gb.GBP_ERR_NAN
    assert not pj.stats.converged
    pj.close()
    # the allocation-free entry point keeps the launched form
    lib, st, prm = gb.load_library(), gb.Stats(), gb.make_params(Residual=1e-6)
    vp = ctypes.c_void_p
    lib.gbp_project_device_static.argtypes = [ctypes.c_int] * 4 + [ctypes.c_double] * 2 + [vp] * 5 + \
        [ctypes.POINTER(gb.Params), vp, ctypes.POINTER(gb.Stats), vp]
    rc = lib.gbp_project_device_static(3, sc.nx, sc.ny, sc.nz, sc.dx, sc.dt, solid.data_ptr(), fluid.data_ptr(),
                                       *(t.data_ptr() for t in other), ctypes.byref(prm), p.data_ptr(),
                                       ctypes.byref(st), vp(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == gb.GBP_ERR_NAN and not st.converged
