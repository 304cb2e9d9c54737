"""The preconditioned solve's direction pass, which forms A p by a recurrence from
A z: in FP64 a product that is not A p would part the recurred residual, the
stopping rule's, from b - A x (drift of the recurrences: about 1e-13 of |b|); in
mixed precision, where the refinement repairs it, it would cost iterations. The
shapes take the plane-by-plane and the four-plane forms (above 64^3 cells), even
and odd rows, clipped tiles and 2D."""
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(12, 10, 9), (31, 17, 13), (66, 65, 64), (130, 49, 43), (65, 66, 67), (50, 34), (65, 9)])
def test_recurred_product(n):
    sc = scenes.liquid2(n, seed=7) if len(n) == 2 else scenes.liquid3(n, seed=7)
    its = {}
    for precision in ("fp64", "mixed"):
        vel = [a.copy() for a in (sc.u, sc.v, sc.w)[: len(n)]]
        pj = gb.projector_for(sc, Residual=1e-8, Solver="mgpcg", Precision=precision)
        assert pj.project(sc.dt, vel, sc.solid, sc.fluid) == gb.GBP_OK
        assert pj.stats.true_resid_inf <= 1.01e-8
        its[precision] = pj.stats.iterations
        pj.close()
    # three inner solves to 1e-3, each from a new direction
    assert its["mixed"] <= 2 * its["fp64"] + 8
