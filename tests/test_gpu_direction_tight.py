"""The preconditioned solve's product by a recurrence, q = A z + beta q, at a tight
residual in FP64: b - A x follows the recurred residual, which the solve stops on,
to 1e-13 of |b| (each iteration's rounding of q and r, below 1e-15 of the vectors'
largest value, over some thirty iterations of vectors up to a few |b|)."""
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["liquid3", "smoke3"])
@pytest.mark.parametrize("n", [(33, 31, 40), (66, 65, 64), (96, 80, 72)])
def test_residual_follows(kind, n):
    sc = getattr(scenes, kind)(n, seed=7)
    pj = gb.projector_for(sc, Residual=1e-12, Solver="mgpcg", Precision="fp64")
    assert pj.project(sc.dt, [a.copy() for a in (sc.u, sc.v, sc.w)], sc.solid, sc.fluid) == gb.GBP_OK
    assert pj.stats.reresid <= 1e-12 and abs(pj.stats.true_resid_inf - pj.stats.reresid) <= 1e-13
    pj.close()
