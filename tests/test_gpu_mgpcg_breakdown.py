"""MGPCG on a right-hand side that holds NaN: GBP_ERR_NAN, not a converged solve
(|r|_inf of nothing but NaN must not count as 0), alone and beside a sound
scene of a batch, whose result is as alone."""
import numpy as np
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("every", [True, False])
@pytest.mark.parametrize("n", [(20, 18, 22), (66, 64, 65)])
def test_nan_velocity(n, every, precision):
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    cfg = dict(Residual=1e-6, Solver="mgpcg", Precision=precision)
    sc = scenes.smoke3(n, seed=2)
    solid, fluid = dev(sc.solid), dev(sc.fluid)

    def velocity(bad):
        vel = [dev(a) for a in (sc.u, sc.v, sc.w)]
        if bad and every:
            vel[0].fill_(np.nan)
        elif bad:
            vel[0][3, 4, 5] = np.nan
        return vel
    pjs = [gb.projector_for(sc, **cfg) for _ in range(2)]
    p, q = (torch.empty(sc.fluid.shape, device="cuda") for _ in range(2))
    assert pjs[0].project(sc.dt, velocity(True), solid, fluid, pressure_out=p) == gb.GBP_ERR_NAN
    assert not pjs[0].stats.converged
    batch = gb.Batch(pjs, **cfg)
    vel = [velocity(True), velocity(False)]
    assert batch.project([sc.dt] * 2, vel, [solid] * 2, [fluid] * 2, [p, q]) == gb.GBP_ERR_NAN
    assert not batch.stats[0].converged and batch.stats[1].converged
    assert batch.stats[1].true_resid_inf <= 1.01e-6 and bool(torch.isfinite(q).all())
    batch.close()
    for pj in pjs:
        pj.close()
