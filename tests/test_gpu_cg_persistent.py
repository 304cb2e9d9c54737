"""The single-launch CG on grids (cg_resident.cu) at the edges of its shapes: a
handful of unknowns, the cluster's largest grid and the cooperative launch's
smallest, one and several unknowns a thread, grids whose unknowns do not fit
(left to the launched form), solves cut off at the iteration limit."""
import ctypes

import numpy as np
import pytest

import oracle
import shiokaze_gb300 as gb
from gpu_util import rel_inf
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("liquid2", (9, 7)), ("liquid2", (128, 128)), ("liquid2", (129, 128)),
                                    ("liquid2", (500, 300)), ("smoke3", (16, 4, 3)), ("liquid3", (33, 8, 64)),
                                    ("smoke3", (25, 26, 26)), ("liquid3", (63, 57, 50)), ("smoke3", (64, 63, 62)),
                                    ("liquid3", (100, 99, 98)), ("smoke3", (90, 92, 95)), ("smoke3", (100, 99, 98))])
def test_first_iterations_match_oracle(kind, n):
    """Three iterations: the same FP64 iterates up to the order of the sums,
    whose rounding CG multiplies by less than ten a step (numpy, 1e-15 to 3e-4
    in thirty), so far below a float's."""
    sc = getattr(scenes, kind)(n, seed=3)
    dim = len(n)
    want = oracle.project_scene(sc, "port", residual=1e-6, max_iterations=3)
    vel = [a.copy() for a in (sc.u, sc.v, sc.w)[:dim]]
    pj = gb.projector_for(sc, Residual=1e-6, MaxIterations=3)
    assert pj.project(sc.dt, vel, sc.solid, sc.fluid) == gb.GBP_ERR_NOT_CONVERGED
    assert pj.stats.iterations == 3
    assert abs(pj.stats.reresid - want.reresid) <= 1e-9 * want.reresid
    assert rel_inf(pj.get_pressure(), want.pressure) <= 1e-6
    for a, b in zip(vel, (want.u, want.v, want.w)):
        assert rel_inf(a, b) <= 1e-6
    pj.close()


@pytest.mark.parametrize("kind,n", [("liquid2", (128, 128)), ("liquid3", (40, 37, 22)), ("smoke3", (48, 40, 44)),
                                    ("smoke3", (5, 3, 2000)), ("liquid3", (75, 92, 61))])
@pytest.mark.parametrize("residual", [1e-4, 1e-6, 1e-10])
def test_converged_residual(kind, n, residual):
    """The recomputed FP64 residual of the solution is what the recurrence
    stopped at (it drifts by the rounding of a thousand updates at most)."""
    sc = getattr(scenes, kind)(n, seed=5)
    vel = [a.copy() for a in (sc.u, sc.v, sc.w)[: len(n)]]
    pj = gb.projector_for(sc, Residual=residual)
    assert pj.project(sc.dt, vel, sc.solid, sc.fluid) == gb.GBP_OK
    assert pj.stats.reresid <= residual
    assert abs(pj.stats.true_resid_inf - pj.stats.reresid) <= 1e-12
    pj.close()


@pytest.mark.parametrize("n", [(24, 20, 18), (32, 32, 32), (40, 37, 22)])
@pytest.mark.parametrize("limit", [1, 40, 30000])
def test_equals_allocation_free_entry(n, limit):
    """Both entry points run the same solve: the same bits."""
    import torch
    sc = scenes.liquid3(n, seed=5)
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
