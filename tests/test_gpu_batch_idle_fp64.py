"""As test_gpu_batch_idle, in FP64: the update launches lower the counter of
unfinished scenes themselves, so blocks of the launch in which the last scene ends
start before and after that."""
import numpy as np
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_small_scenes_repeated_fp64():
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    scs = [scenes.liquid3(n, seed=n) for n in (34, 35, 37, 39, 43, 44, 47, 48, 51, 52, 55, 57, 58, 69, 71, 72)]
    cfg = dict(Residual=1e-6, Solver="mgpcg", Precision="fp64")
    pjs = [gb.projector_for(sc, **cfg) for sc in scs]
    batch = gb.Batch(pjs, **cfg)
    solid, fluid = [dev(sc.solid) for sc in scs], [dev(sc.fluid) for sc in scs]
    first = None
    for _ in range(12):
        vel = [[dev(a) for a in (sc.u, sc.v, sc.w)] for sc in scs]
        p = [torch.empty(sc.fluid.shape, device="cuda") for sc in scs]
        assert batch.project([sc.dt for sc in scs], vel, solid, fluid, p) == gb.GBP_OK
        first = first or [t.clone() for t in p]
        assert all(torch.equal(a, b) for a, b in zip(p, first))
    batch.close()
    for pj in pjs:
        pj.close()
