"""A batched scene's result does not depend on the other scenes of its batch: the
same bits in a small batch, in a large one (whose list of tiles is dealt to the
blocks in groups) and anywhere in it; for scenes of at most one item a block
(64^3 and less on this GPU) also alone."""
import numpy as np
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


def _solve(scs, precision):
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    cfg = dict(Residual=1e-6, Solver="mgpcg", Precision=precision)
    pjs = [gb.projector_for(sc, **cfg) for sc in scs]
    batch = gb.Batch(pjs, **cfg)
    vel = [[dev(a) for a in (sc.u, sc.v, sc.w) if a is not None] for sc in scs]
    p = [torch.empty(sc.fluid.shape, device="cuda") for sc in scs]
    assert batch.project([sc.dt for sc in scs], vel, [dev(sc.solid) for sc in scs], [dev(sc.fluid) for sc in scs],
                         p) == gb.GBP_OK
    torch.cuda.synchronize()
    out = [([a.view(torch.int32) for a in (q, *v)], (s.iterations, s.true_resid_inf, s.true_resid_l2))
           for q, v, s in zip(p, vel, batch.stats)]
    batch.close()
    for pj in pjs:
        pj.close()
    return out


def _same(a, b):
    import torch
    return a[1] == b[1] and all(torch.equal(x, y) for x, y in zip(a[0], b[0]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_same_in_any_company(precision):
    small = [scenes.liquid3((40, 33, 37), seed=1), scenes.smoke3((31, 30, 29), seed=2), scenes.liquid2((70, 66), seed=3)]
    large = scenes.liquid3((101, 100, 99), seed=4)
    others = [scenes.liquid3(64, seed=10 + k) for k in range(24)]
    few = _solve([others[0], *small, large], precision)
    many = _solve([*others[:9], *small[::-1], *others[9:17], large, *others[17:]], precision)
    more = _solve([large, *others, *others, *small], precision)
    for k, sc in enumerate(small):
        assert _same(few[1 + k], many[9 + 2 - k]) and _same(few[1 + k], more[-3 + k]), sc.name
        assert _same(few[1 + k], _solve([sc], precision)[0]), sc.name
    assert _same(few[0], many[0]) and _same(few[0], more[1]) and _same(few[0], _solve([others[0]], precision)[0])
    assert _same(few[4], many[20]) and _same(few[4], more[0]), "large"
