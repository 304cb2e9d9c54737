"""Blocks of the refinement and update launches that start while the last scene
that needs them ends: a batch of many small scenes that converge at different
iterations, solved again and again, gives the same bits each time."""
import numpy as np
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_small_scenes_repeated():
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    scs = [scenes.liquid3(n, seed=n) for n in (34, 35, 37, 39, 43, 44, 47, 48, 51, 52, 55, 57, 58, 69, 71, 72)]
    cfg = dict(Residual=1e-6, Solver="mgpcg", Precision="mixed")
    pjs = [gb.projector_for(sc, **cfg) for sc in scs]
    batch = gb.Batch(pjs, **cfg)
    solid, fluid = [dev(sc.solid) for sc in scs], [dev(sc.fluid) for sc in scs]
    first = None
    for _ in range(12):
        vel = [[dev(a) for a in (sc.u, sc.v, sc.w)] for sc in scs]
        p = [torch.empty(sc.fluid.shape, device="cuda") for sc in scs]
        batch.project([sc.dt for sc in scs], vel, solid, fluid, p)
        first = first or [t.clone() for t in p]
        assert all(torch.equal(a, b) for a, b in zip(p, first))
