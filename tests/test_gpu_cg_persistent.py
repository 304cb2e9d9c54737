"""The single-launch CG (cg_persistent.cuh) at the edges of its shapes: one
virtual block, the cluster's largest grid and the cooperative grid's smallest,
several virtual blocks side by side and in rounds, several tiles a thread (long
thin grids have many tiles of few cells). It equals the allocation-free entry
point, which keeps the launched form, bit for bit, also when the iteration
limit cuts the solve off."""
import ctypes

import numpy as np
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("liquid3", (9, 7, 1)), ("liquid3", (32, 8, 64)), ("liquid3", (33, 8, 33)),
                                    ("liquid3", (32, 32, 32)), ("liquid3", (40, 37, 22)), ("smoke3", (2, 9, 300)),
                                    ("smoke3", (5, 3, 2000)), ("smoke3", (2, 2, 8000))])
@pytest.mark.parametrize("limit", [1, 40, 400])
def test_equals_launched_form(kind, n, limit):
    import torch
    sc = getattr(scenes, kind)(n, seed=5)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    solid, fluid = dev(sc.solid), dev(sc.fluid)
    a, b = ([dev(x) for x in (sc.u, sc.v, sc.w)] for _ in range(2))
    pa, pb = (torch.empty(sc.fluid.shape, device="cuda") for _ in range(2))
    pj = gb.projector_for(sc, Residual=1e-6, MaxIterations=limit)
    ra = pj.project(sc.dt, a, solid, fluid, pressure_out=pa)
    lib = gb.load_library()
    st, prm = gb.Stats(), gb.make_params(Residual=1e-6, MaxIterations=limit)
    vp = ctypes.c_void_p
    lib.gbp_project_device_static.argtypes = [ctypes.c_int] * 4 + [ctypes.c_double] * 2 + [vp] * 5 + \
        [ctypes.POINTER(gb.Params), vp, ctypes.POINTER(gb.Stats), vp]
    torch.cuda.synchronize()
    rb = lib.gbp_project_device_static(3, sc.nx, sc.ny, sc.nz, sc.dx, sc.dt, solid.data_ptr(), fluid.data_ptr(),
                                       *(t.data_ptr() for t in b), ctypes.byref(prm), pb.data_ptr(), ctypes.byref(st),
                                       vp(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert ra == rb and pj.stats.iterations == st.iterations
    for x, y in zip([pa, *a], [pb, *b]):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32))
    pj.close()
