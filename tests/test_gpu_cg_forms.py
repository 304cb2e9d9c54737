"""The forms of plain CG: one launch in a cluster (up to 64 blocks of 256 rows), one
launch over all SMs, and launched iterations. The one-launch form's waits between
blocks are bounded: gbp_debug_cg makes them run out (one block leaves out its
arrivals, as a block that stopped would; nothing faults), the solve returns
GBP_ERR_CUDA and the next one on the same context is normal. The forms agree bit
for bit, also where the one-launch form is resumed by another launch."""
import ctypes

import numpy as np
import pytest

import shiokaze_gb300 as gb
from shiokaze_gb300 import scenes

pytestmark = pytest.mark.gpu


def _debug(pj=None, launched=0, steps=0, block=0, polls=0):
    lib, ctx = gb.load_library(), gb.default_context()
    lib.gbp_debug_cg.argtypes = [ctypes.c_void_p, ctypes.c_void_p] + [ctypes.c_int] * 4
    return lib.gbp_debug_cg(ctx.handle, pj.scene if pj else None, launched, steps, block, polls)


def _rows(n):
    """A symmetric tridiagonal matrix with a far diagonal, and a right-hand side."""
    rng = np.random.default_rng(n)
    far = n // 2
    near, away = rng.random(n - 1) + 0.5, rng.random(n - far) + 0.5
    d = np.full(n, 0.01)
    d[:-1] += near
    d[1:] += near
    d[:-far] += away
    d[far:] += away
    r = np.concatenate([np.arange(n), np.arange(n - 1), np.arange(1, n), np.arange(n - far), np.arange(far, n)])
    c = np.concatenate([np.arange(n), np.arange(1, n), np.arange(n - 1), np.arange(far, n), np.arange(n - far)])
    v = np.concatenate([d, -near, -near, -away, -away])
    o = np.lexsort((c, r))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))])
    return ptr, c[o], v[o], rng.standard_normal(n)


def _same(a, b):
    return np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).view(np.uint8))


@pytest.mark.parametrize("block", [0, 70])
def test_rows_wait_runs_out(block):
    m = _rows(20000)
    x0, rc0, st0 = gb.csr_cg(*m, residual=1e-9, max_iterations=40)
    assert _debug(block=block, polls=256) == gb.GBP_OK
    with pytest.raises(gb.GBPError) as err:
        gb.csr_cg(*m, residual=1e-9, max_iterations=40)
    assert err.value.code == gb.GBP_ERR_CUDA and "wait between the blocks" in str(err.value)
    x1, rc1, st1 = gb.csr_cg(*m, residual=1e-9, max_iterations=40)
    assert rc0 == rc1 and st0["iterations"] == st1["iterations"] and _same(x0, x1)


@pytest.mark.parametrize("block", [0, 100])
def test_grid_wait_runs_out(block):
    sc = scenes.liquid3((40, 37, 22), seed=5)
    pj = gb.projector_for(sc, Residual=1e-6)

    def solve():
        vel = tuple(a.copy() for a in (sc.u, sc.v, sc.w))
        return pj.project(sc.dt, vel, sc.solid, sc.fluid), pj.get_pressure().copy(), vel
    want = solve()
    assert _debug(pj, block=block, polls=256) == gb.GBP_OK
    with pytest.raises(gb.GBPError) as err:
        solve()
    assert err.value.code == gb.GBP_ERR_CUDA and "wait between the blocks" in str(err.value)
    got = solve()
    assert got[0] == want[0] == gb.GBP_OK and _same(got[1], want[1])
    assert all(_same(a, b) for a, b in zip(got[2], want[2]))
    pj.close()


def test_bad_arguments():
    for kw in (dict(steps=-1), dict(block=-1), dict(polls=-1), dict(polls=(1 << 22) + 1)):
        assert _debug(**kw) == gb.GBP_ERR_INVALID_ARGUMENT


# one virtual block, the cluster's last row count and the next, a row more
# than one a thread of the launched grid, several rows a thread
@pytest.mark.parametrize("n", [200, 16384, 16385, 233473, 300001])
def test_rows_forms_agree(n):
    m = _rows(n)
    x0, rc0, st0 = gb.csr_cg(*m, residual=1e-9, max_iterations=30)
    assert _debug(launched=1) == gb.GBP_OK
    x1, rc1, st1 = gb.csr_cg(*m, residual=1e-9, max_iterations=30)
    assert rc0 == rc1 and st0["iterations"] == st1["iterations"] and _same(x0, x1)


@pytest.mark.parametrize("n", [200, 20000])
@pytest.mark.parametrize("limit,steps", [(30, 7), (28, 7), (5, 7)])
def test_rows_resumed(n, limit, steps):
    m = _rows(n)
    x0, rc0, st0 = gb.csr_cg(*m, residual=1e-9, max_iterations=limit)
    assert _debug(steps=steps) == gb.GBP_OK
    x1, rc1, st1 = gb.csr_cg(*m, residual=1e-9, max_iterations=limit)
    assert rc0 == rc1 and st0["iterations"] == st1["iterations"] and _same(x0, x1)


@pytest.mark.parametrize("n", [(9, 7, 1), (40, 37, 22)])
@pytest.mark.parametrize("limit,kw", [(400, dict(steps=7)), (21, dict(steps=7)), (400, dict(launched=1))])
def test_grid_forms_agree(n, limit, kw):
    sc = scenes.liquid3(n, seed=5)
    pj = gb.projector_for(sc, Residual=1e-6, MaxIterations=limit)

    def solve():
        vel = tuple(a.copy() for a in (sc.u, sc.v, sc.w))
        return pj.project(sc.dt, vel, sc.solid, sc.fluid), pj.stats.iterations, pj.get_pressure().copy(), vel
    want = solve()
    assert _debug(pj, **kw) == gb.GBP_OK
    got = solve()
    assert got[:2] == want[:2] and _same(got[2], want[2]) and all(_same(a, b) for a, b in zip(got[3], want[3]))
    pj.close()
