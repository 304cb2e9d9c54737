"""The one-block tail of the multigrid cycle at the shapes where its coarsest
level changes form: a matrix for at most 64 cells (one warp's slots), sweeps
beyond, single cells and rows, in 2D and 3D, all-fluid (singular) systems among
them. A preconditioner that is not the fixed symmetric operator it should be
shows in the iterations; the solve's own FP64 residual is its stopping rule."""
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 8, 8), (7, 7, 7), (16, 4, 2), (24, 24, 24), (28, 20, 9), (33, 31, 17), (16, 16),
                               (28, 12), (100, 7)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_coarsest_forms(n, precision):
    sc = scenes.liquid2(n, seed=4) if len(n) == 2 else scenes.liquid3(n, seed=4)
    vel = [a.copy() for a in (sc.u, sc.v, sc.w)[: len(n)]]
    pj = gb.projector_for(sc, Residual=1e-6, Solver="mgpcg", Precision=precision)
    assert pj.project(sc.dt, vel, sc.solid, sc.fluid) == gb.GBP_OK
    assert pj.stats.true_resid_inf <= 1.01e-6
    assert pj.stats.iterations <= 40
    pj.close()
