"""The steps after a projection where their kernels can go wrong, against the
oracle bit for bit: extrapolation with rows and planes that are no multiple of
the four cells a thread takes, single rows and cells, no round, one round, more
rounds than a byte counts; the solid constraint with everything, nothing and
scattered faces inside the solid, near-zero levels and values at the float
range's lower end."""
import numpy as np
import pytest

import oracle
import shiokaze_gb300 as gb

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    """Equal bits; any NaN equals any NaN."""
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(a)
    return np.array_equal(nan, np.isnan(b)) and np.array_equal(a.view(np.uint32)[~nan], b.view(np.uint32)[~nan])


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 9), (2, 3, 5), (7, 1, 4), (3, 2, 33), (5, 6, 64), (20, 19, 21)])
@pytest.mark.parametrize("count", [0, 1, 2, 7, 260])
def test_extrapolate(shape, count):
    import torch
    rng = np.random.default_rng(sum(shape) + count)
    a = rng.normal(0, 1, shape).astype(np.float32)
    m = (rng.random(shape) < (0.02 if a.size > 500 else 0.2)).astype(np.uint8)
    m.flat[rng.integers(0, m.size)] = 1
    want, wm, added = oracle.extrapolate3(a, m, count)
    util = gb.MacUtility3(2, 2, 2, 0.5)
    d, dm = torch.from_numpy(a.copy()).cuda(), torch.from_numpy(m.copy()).cuda()
    assert util.extrapolate(d, dm, count) == added
    assert np.array_equal(dm.cpu().numpy(), wm)
    # the oracle reads inactive cells as 0, the call leaves their values alone
    got = d.cpu().numpy()
    assert same_bits(np.where(wm != 0, got, np.float32(0)), want)
    assert same_bits(got[wm == 0], a[wm == 0])


@pytest.mark.parametrize("n,kind", [((2, 2, 2), "all"), ((2, 3, 2), "some"), ((9, 4, 35), "some"), ((33, 17, 6), "some"),
                                    ((33, 17, 6), "none"), ((20, 9, 11), "hair"), ((12, 10, 14), "tiny"),
                                    ((18, 16, 7), "odd")])
@pytest.mark.parametrize("dx", [1.0 / 32, 0.013])
def test_constrain(n, kind, dx):
    import torch
    nx, ny, nz = n
    rng = np.random.default_rng(nx * ny + nz)
    solid = rng.normal(0, dx, (nz + 1, ny + 1, nx + 1))
    if kind in ("all", "none"):
        solid = np.abs(solid) * (-1 if kind == "all" else 1)
    elif kind == "hair":
        solid *= 10.0 ** rng.uniform(-9, 0, solid.shape)
    solid = solid.astype(np.float32)
    if kind == "tiny":
        solid *= (2.0 ** rng.uniform(-130, 0, solid.shape)).astype(np.float32)
    shapes = [(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)]
    vel = [rng.normal(0, 1, s).astype(np.float32) for s in shapes]
    if kind == "tiny":
        vel = [v * (2.0 ** rng.uniform(-140, 0, v.shape)).astype(np.float32) for v in vel]
    if kind == "odd":
        solid.flat[rng.integers(0, solid.size, 3)] = [np.nan, np.inf, -np.inf]
        vel[0].flat[rng.integers(0, vel[0].size, 2)] = [np.nan, np.inf]
    masks = [(rng.random(s) < 0.8).astype(np.uint8) for s in shapes]
    vel = [np.where(m != 0, v, np.float32(0)) for v, m in zip(vel, masks)]
    util = gb.MacUtility3(nx, ny, nz, dx)
    for ms in (masks, [None] * 3):
        want = oracle.constrain3(solid, *vel, dx, masks=ms)
        got = [torch.from_numpy(v.copy()).cuda() for v in vel]
        util.constrain_velocity(torch.from_numpy(solid).cuda(), tuple(got),
                                None if ms[0] is None else [torch.from_numpy(m).cuda() for m in ms])
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert same_bits(g.cpu().numpy(), w)
