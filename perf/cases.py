"""Performance cases of the GB300 projection, advection and velocity utilities.

Each case is one call sequence that a simulation runs every time step, through
the Python mirror of the C ABI (``shiokaze_gb300``):

* ``project``  ``MacProject2`` / ``MacProject3.project`` on device arrays
* ``bricks``   ``MacProject3.project_bricks`` on host arrays, the call that the
               plugin module makes with the reference's sparse arrays
* ``batch``    ``Batch.project``: independent liquid scenes of uneven sizes
* ``served``   three ticks of a server: resident liquid and smoke scenes, one
               warm-started batched projection per tick
* ``advect``   ``MacAdvection2`` / ``MacAdvection3.advect_step`` (MacCormack)
* ``after``    ``MacUtility3``: extrapolation of the three components and the
               solid constraint, the steps after a liquid projection
* ``csr``      ``csr_cg``, the linear-solver module's call on host arrays

``listed()`` names twelve of them, ``draw(rng)`` gives others of the same
ranges. ``exact()`` computes the same results in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import shiokaze_gb300 as gb

DEV = "cuda"
DT = 1.0 / 60.0
GRAVITY = -9.8
RESIDUAL = 1e-6
EPS = 1e-2  # EpsSolid and EpsFluid, the reference's defaults
F64 = torch.float64


# --------------------------------------------------------------------------
# the cases


def listed():
    return [
        # the smallest call: a 2D liquid step with the reference's plain CG in
        # FP64, where launches and the host's polls count
        {"name": "plane_liquid_128_cg", "kind": "project", "scene": "liquid", "dim": 2, "nx": 128, "ny": 128, "nz": 1,
         "solver": "cg", "precision": "fp64"},
        # the smallest 3D scene that the server admits
        {"name": "liquid_32_mixed", "kind": "project", "scene": "liquid", "dim": 3, "nx": 32, "ny": 32, "nz": 32,
         "solver": "mgpcg", "precision": "mixed"},
        # the reference's default solver (plain CG, FP64) on a ragged 3D grid
        {"name": "liquid_75x92x61_cg", "kind": "project", "scene": "liquid", "dim": 3, "nx": 75, "ny": 92, "nz": 61,
         "solver": "cg", "precision": "fp64"},
        # the plugin's boundary: a 128^3 liquid in sparse bricks on the host
        {"name": "bricks_liquid_128_mixed", "kind": "bricks", "scene": "liquid", "dim": 3, "nx": 128, "ny": 128,
         "nz": 128, "solver": "mgpcg", "precision": "mixed"},
        # the headline workload, 256^3 smoke, in both precisions
        {"name": "smoke_256_mixed", "kind": "project", "scene": "smoke", "dim": 3, "nx": 256, "ny": 256, "nz": 256,
         "solver": "mgpcg", "precision": "mixed"},
        {"name": "smoke_256_fp64", "kind": "project", "scene": "smoke", "dim": 3, "nx": 256, "ny": 256, "nz": 256,
         "solver": "mgpcg", "precision": "fp64"},
        # the batched workload: 64 liquids, edges log-uniform in [32, 160]
        {"name": "batch_64_mixed", "kind": "batch", "count": 64, "lo": 32, "hi": 160, "mix": 4,
         "precision": "mixed"},
        # a server's ticks over scenes of its usual sizes, warm-started
        {"name": "served_6_mixed", "kind": "served", "count": 6, "lo": 32, "hi": 128, "mix": 5,
         "precision": "mixed"},
        # one advection step of the 256^3 smoke: density, then velocity
        {"name": "advect_smoke_256", "kind": "advect", "scene": "smoke", "dim": 3, "nx": 256, "ny": 256, "nz": 256},
        # the 2D advection of a liquid's level set and velocity, ragged
        {"name": "advect_plane_liquid_1000x777", "kind": "advect", "scene": "liquid", "dim": 2, "nx": 1000, "ny": 777,
         "nz": 1},
        # the velocity steps after a liquid projection, ragged
        {"name": "after_liquid_150x131x170", "kind": "after", "nx": 150, "ny": 131, "nz": 170, "width": 3},
        # a pressure matrix through the linear-solver module
        {"name": "csr_liquid_64", "kind": "csr", "nx": 64, "ny": 64, "nz": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edges3(rng, lo, hi, most):
    """Three edges near each other, odd ones among them, of at most `most` cells."""
    n = _log_int(rng, lo, hi)
    if rng.random() < 0.3:
        return (n, n, n)
    e = [max(lo, min(hi, int(n * rng.uniform(0.7, 1.3)))) for _ in range(3)]
    while e[0] * e[1] * e[2] > most:
        e = [max(lo, int(0.95 * x)) for x in e]
    return tuple(e)


def draw(rng: random.Random):
    kind = rng.choice(["project", "project", "project", "bricks", "batch", "served", "advect", "advect", "after", "csr"])
    scene = rng.choice(["liquid", "smoke"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "project":
        solver = rng.choice(["cg", "mgpcg", "mgpcg"])
        if rng.random() < 0.25:
            nx, ny, nz, dim = _log_int(rng, 48, 320), _log_int(rng, 48, 320), 1, 2
        else:
            dim = 3
            nx, ny, nz = _edges3(rng, 24, 112, 112 ** 3) if solver == "cg" else _edges3(rng, 24, 256, 256 ** 3)
        return {"kind": "project", "scene": scene, "dim": dim, "nx": nx, "ny": ny, "nz": nz, "solver": solver,
                "precision": "fp64" if solver == "cg" else precision}
    if kind == "bricks":
        nx, ny, nz = _edges3(rng, 32, 128, 128 ** 3)
        return {"kind": "bricks", "scene": scene, "dim": 3, "nx": nx, "ny": ny, "nz": nz, "solver": "mgpcg",
                "precision": precision}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(8, 48), "lo": 32, "hi": _log_int(rng, 64, 160),
                "mix": rng.randrange(1 << 20), "precision": precision}
    if kind == "served":
        return {"kind": "served", "count": rng.randint(2, 10), "lo": 32, "hi": _log_int(rng, 48, 128),
                "mix": rng.randrange(1 << 20), "precision": precision}
    if kind == "advect":
        if rng.random() < 0.3:
            return {"kind": "advect", "scene": scene, "dim": 2, "nx": _log_int(rng, 64, 1400),
                    "ny": _log_int(rng, 64, 1400), "nz": 1}
        nx, ny, nz = _edges3(rng, 24, 256, 256 ** 3)
        return {"kind": "advect", "scene": scene, "dim": 3, "nx": nx, "ny": ny, "nz": nz}
    if kind == "after":
        nx, ny, nz = _edges3(rng, 24, 256, 256 ** 3)
        return {"kind": "after", "nx": nx, "ny": ny, "nz": nz, "width": rng.randint(1, 5)}
    nx, ny, nz = _edges3(rng, 20, 72, 72 ** 3)
    return {"kind": "csr", "nx": nx, "ny": ny, "nz": nz}


# --------------------------------------------------------------------------
# scenes on the GPU: the liquid and smoke shapes of shiokaze_gb300.scenes,
# with their geometry moved a little by the seed


class _Scene:
    def __init__(self, dim, nx, ny, nz):
        self.dim, self.nx, self.ny, self.nz = dim, nx, ny, nz
        self.dx = 1.0 / max(nx, ny, nz)


def _axes(sc, shape, offs):
    """Coordinates of a (z, y, x) grid with the per-axis offsets in cells."""
    x, y, z = ((torch.arange(n, dtype=F64, device=DEV) + o) * sc.dx for n, o in zip(shape[::-1], offs))
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _ball(x, y, z, c, r, dim):
    d = (x - c[0]) ** 2 + (y - c[1]) ** 2
    return torch.sqrt(d + (z - c[2]) ** 2 if dim == 3 else d + 0 * z) - r


def _band(phi, dx):
    """A narrow-band level set read densely: exact within sqrt(3) dx."""
    half = math.sqrt(3.0) * dx
    b = np.float32(half).item()
    return torch.where(phi.abs() < half, phi.float(), torch.where(phi < 0, -b, b)).float().contiguous()


def _shapes(sc):
    """(z, y, x) shapes of the nodes, the cells and the face components."""
    nx, ny, nz = sc.nx, sc.ny, sc.nz
    nodes = (nz + 1 if sc.dim == 3 else 1, ny + 1, nx + 1)
    faces = [(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)][: sc.dim]
    return nodes, (nz, ny, nx), faces


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _make_scene(kind, dim, nx, ny, nz, seed, pool=None, still=False):
    """Level sets, and velocities as the step before a projection leaves them:
    noise, and gravity over one step for a liquid. A `still` scene's geometry
    is the same for every seed: where the number of outputs depends on it."""
    sc = _Scene(dim, nx, ny, nz)
    rng, g = random.Random(11 if still else int(seed)), _generator(seed)
    nodes, cells, faces = _shapes(sc)
    nx_, ny_, nz_ = (n * sc.dx for n in (nx, ny, nz))  # the domain's extent
    xn, yn, zn = _axes(sc, nodes, (0, 0, 0))
    xc, yc, zc = _axes(sc, cells, (0.5, 0.5, 0.5))
    if kind == "liquid":
        c = (nx_ * rng.uniform(0.4, 0.6), ny_ * rng.uniform(0.7, 0.8), nz_ * rng.uniform(0.4, 0.6))
        small = min(nx_, ny_, nz_) if dim == 3 else min(nx_, ny_)
        level = ny_ * (rng.uniform(0.3, 0.4) if pool is None else pool)
        sc.phi = torch.minimum(yc - level + 0 * xc + 0 * zc, _ball(xc, yc, zc, c, 0.16 * small, dim))
        if dim == 3:  # a static sphere in the pool
            s = (nx_ * rng.uniform(0.4, 0.6), 0.2 * ny_, nz_ * rng.uniform(0.4, 0.6))
            sc.solid_phi = _ball(xn, yn, zn, s, 0.12 * small, 3)
            sc.phi = torch.maximum(sc.phi, -(_ball(xc, yc, zc, s, 0.12 * small, 3) + sc.dx))
        else:
            sc.solid_phi = torch.full(nodes, 1.0, dtype=F64, device=DEV)
        sc.fluid, sigma = _band(sc.phi, sc.dx), 0.2
    else:
        c = (nx_ * rng.uniform(0.4, 0.6), ny_ * rng.uniform(0.4, 0.6), 0.0)
        sc.solid_phi = _ball(xn, yn, zn, c, 0.1 * min(nx_, ny_), 2)
        sc.phi = torch.full(cells, -1.0, dtype=F64, device=DEV)
        sc.fluid, sigma = sc.phi.float(), 1.0
    sc.solid = _band(sc.solid_phi, sc.dx)
    sc.vel = [sigma * torch.randn(s, generator=g, device=DEV) for s in faces]
    if kind == "liquid":
        sc.vel[1] += GRAVITY * DT
    return sc


def _of_case(case, seed):
    return _make_scene(case["scene"], case["dim"], case["nx"], case["ny"], case["nz"], seed,
                       still=case["kind"] == "bricks")


def _csr_scene(case, seed):
    return _make_scene("liquid", 3, case["nx"], case["ny"], case["nz"], seed, still=True)


def _mixed_scenes(case, seed):
    """The scenes of a batch or a server: sizes from the case, the rest from the seed."""
    sizes, out = random.Random(int(case["mix"])), []
    for n in range(case["count"]):
        edge = _log_int(sizes, case["lo"], case["hi"])
        kind = "liquid" if case["kind"] == "batch" or sizes.random() < 0.7 else "smoke"
        pool = sizes.uniform(0.1, 0.6) if case["kind"] == "batch" else None
        out.append(_make_scene(kind, 3, edge, edge, edge, int(seed) * 1009 + n, pool))
        out[-1].smoke = kind == "smoke"
    return out


def _near_liquid(sc, d, width):
    """Faces of component d within `width` cells of the liquid: a liquid's active faces."""
    a = sc.phi
    lo = torch.nn.functional.pad(a, _pad1(d, 1, 0), value=math.inf)
    hi = torch.nn.functional.pad(a, _pad1(d, 0, 1), value=math.inf)
    return torch.minimum(lo, hi) < width * sc.dx


def _pad1(d, before, after):
    p = [0] * 6
    p[2 * d], p[2 * d + 1] = before, after
    return p


def _flow(sc, seed, sigma):
    """A smooth swirling flow that stops at the walls, of a few cells a step, with a little noise."""
    rng, g = random.Random(int(seed) + 99), _generator(seed + 1)
    speed, out = 3.0 * sc.dx / DT, []
    for d, shape in enumerate(_shapes(sc)[2]):
        offs = [0.5, 0.5, 0.5]
        offs[d] = 0.0
        x, y, z = _axes(sc, shape, offs)
        f = torch.zeros(shape, dtype=F64, device=DEV)
        for _ in range(3):
            k = [2 * math.pi * rng.choice([1, 2, 3]) for _ in range(3)]
            ph = [rng.uniform(0, 2 * math.pi) for _ in range(3)]
            zz = torch.sin(k[2] * z + ph[2]) if sc.dim == 3 else 1.0 + 0 * z
            f += rng.uniform(0.3, 0.6) * torch.sin(k[0] * x + ph[0]) * torch.sin(k[1] * y + ph[1]) * zz
        n = (sc.nx, sc.ny, sc.nz)[d] * sc.dx
        f *= torch.sin(math.pi * (x, y, z)[d] / n)
        noise = torch.randn(shape, generator=g, device=DEV)
        out.append((speed * (f.float() + sigma * noise)).contiguous())
    return out


# --------------------------------------------------------------------------
# prepare and run


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("project", "bricks", "csr"):
        cfg = dict(Residual=RESIDUAL, Solver=case.get("solver", "cg"), Precision=case.get("precision", "fp64"))
    if kind == "project":
        sc = _of_case(case, seed)
        st.update(sc=sc, vel=[torch.empty_like(t) for t in sc.vel], pj=gb.projector_for(sc, **cfg),
                  p=torch.empty(_shapes(sc)[1], device=DEV))
    elif kind == "bricks":
        sc = _of_case(case, seed)
        st["pj"] = gb.projector_for(sc, **cfg)
        st["solid"], st["fluid"], st["vel"], st["slots"], _ = _bricks_of(sc)
        st["out"] = None
    elif kind in ("batch", "served"):
        scs = _mixed_scenes(case, seed)
        cfg = dict(Residual=RESIDUAL, Solver="mgpcg", Precision=case["precision"],
                   WarmStart=1 if kind == "served" else 0)
        pjs = [gb.projector_for(sc, **cfg) for sc in scs]
        st.update(scs=scs, pjs=pjs, batch=gb.Batch(pjs, **cfg), vel=[[torch.empty_like(t) for t in sc.vel] for sc in scs],
                  p=[torch.empty(_shapes(sc)[1], device=DEV) for sc in scs])
        if kind == "served":
            st["noise"] = _tick_noise(scs, seed)
    elif kind == "advect":
        sc, q = _advect_inputs(case, seed)
        if case["dim"] == 3:
            adv = gb.MacAdvection3(sc.nx, sc.ny, sc.nz, sc.dx)
        else:
            adv = gb.MacAdvection2(sc.nx, sc.ny, sc.dx)
        st.update(sc=sc, q0=q, q=torch.empty_like(q), vel=[torch.empty_like(t) for t in sc.vel], adv=adv)
    elif kind == "after":
        sc, masks = _after_inputs(case, seed)
        st.update(sc=sc, masks=masks, vel=[torch.empty_like(t) for t in sc.vel],
                  on=[torch.empty_like(m) for m in masks], util=gb.MacUtility3(sc.nx, sc.ny, sc.nz, sc.dx))
    elif kind == "csr":
        st["csr"] = _csr_inputs(case, seed)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "project":
        sc, vel = st["sc"], st["vel"]
        for w, t in zip(vel, sc.vel):
            w.copy_(t)
        st["pj"].project(DT, vel, sc.solid, sc.fluid, pressure_out=st["p"])
        return {"pressure": st["p"], "velocity": vel}
    if kind == "bricks":
        _, st["out"] = st["pj"].project_bricks(DT, st["solid"], st["fluid"], st["vel"], st["slots"], outputs=st["out"])
        return [[v, a] for v, a in st["out"]]
    if kind in ("batch", "served"):
        scs, vel = st["scs"], st["vel"]
        for sc, ws in zip(scs, vel):
            for w, t in zip(ws, sc.vel):
                w.copy_(t)
        for tick in range(1 if kind == "batch" else 3):
            if tick:
                for ws, noise in zip(vel, st["noise"]):
                    for w, t in zip(ws, noise[tick - 1]):
                        w.add_(t)
            st["batch"].project([DT] * len(scs), vel, [sc.solid for sc in scs], [sc.fluid for sc in scs], st["p"])
        # one array per component over the scenes
        return {"pressure": torch.cat([p.reshape(-1) for p in st["p"]]),
                "velocity": [torch.cat([ws[d].reshape(-1) for ws in vel]) for d in range(3)]}
    if kind == "advect":
        sc, vel, q = st["sc"], st["vel"], st["q"]
        q.copy_(st["q0"])
        for w, t in zip(vel, sc.vel):
            w.copy_(t)
        st["adv"].advect_step(tuple(vel), sc.fluid, DT, scalar=q)
        return {"scalar": q, "velocity": vel}
    if kind == "after":
        sc, vel, on = st["sc"], st["vel"], st["on"]
        for d in range(3):
            vel[d].copy_(sc.vel[d])
            on[d].copy_(st["masks"][d])
        for d in range(3):
            st["util"].extrapolate(vel[d], on[d], case["width"])
        st["util"].constrain_velocity(sc.solid, tuple(vel), tuple(on))
        return {"velocity": vel, "active": on}
    indptr, indices, data, b = st["csr"]
    return gb.csr_cg(indptr, indices, data, b, residual=RESIDUAL)[0]


def _tick_noise(scs, seed):
    """What the rest of a time step does to the projected velocity, two ticks of it."""
    g, out = _generator(seed + 5), []
    for sc in scs:
        ticks = []
        for _ in range(2):
            n = [0.05 * torch.randn(t.shape, generator=g, device=DEV) for t in sc.vel]
            n[1] += GRAVITY * DT
            ticks.append(n)
        out.append(ticks)
    return out


def _advect_inputs(case, seed):
    """A smoke's density, or a liquid's level set, and the flow that carries it."""
    sc = _of_case(case, seed)
    sc.vel = _flow(sc, seed, 0.02)
    if case["scene"] == "liquid":
        return sc, sc.fluid.clone()
    x, y, z = _axes(sc, _shapes(sc)[1], (0.5, 0.5, 0.5))
    rng = random.Random(int(seed) + 3)
    c = [rng.uniform(0.3, 0.7) * n * sc.dx for n in (sc.nx, sc.ny, sc.nz)]
    r = 0.3 * min(n for n in (sc.nx, sc.ny, sc.nz) if n > 1) * sc.dx
    q = (1.0 - _ball(x, y, z, c, 0.0, sc.dim) / r).clamp(min=0.0)
    return sc, q.float().contiguous()


def _after_inputs(case, seed):
    """The projected velocity of a liquid: zero off its active faces."""
    sc = _make_scene("liquid", 3, case["nx"], case["ny"], case["nz"], seed)
    vel = _flow(sc, seed, 0.02)
    masks = [_near_liquid(sc, d, 0.0).to(torch.uint8).contiguous() for d in range(3)]
    sc.vel = [(v * m).contiguous() for v, m in zip(vel, masks)]
    return sc, masks


def _bricks_of(sc):
    """The arrays in bricks as the plugin lists them, and the dense velocity
    that they stand for."""
    b = np.float32(math.sqrt(3.0) * sc.dx).item()

    def level(phi, dense):
        a = phi.cpu().numpy()
        half = math.sqrt(3.0) * sc.dx
        return gb.to_bricks(dense.cpu().numpy(), np.abs(a) < half, a <= -half, background=b, fill=-b)[0]

    solid = level(sc.solid_phi + 0 * sc.solid, sc.solid)
    if bool((sc.phi == -1.0).all()):  # a smoke's fluid: filled everywhere, nothing stored
        none = np.zeros(sc.fluid.shape, bool)
        fluid = gb.to_bricks(sc.fluid.cpu().numpy(), none, ~none, background=-1.0, fill=-1.0)[0]
    else:
        fluid = level(sc.phi, sc.fluid)
    vel, dense = [], []
    for d, t in enumerate(sc.vel):
        v, a = gb.to_bricks(t.cpu().numpy(), _near_liquid(sc, d, 3.0).cpu().numpy(), None, background=0.0)
        vel.append(v)
        dense.append(torch.from_numpy(a).to(DEV))
    wet = (fluid[0] >= 0) | ((fluid[0] == gb.BRICK_FILL) & (fluid[3] < 0)) | ((fluid[0] == gb.BRICK_BACKGROUND) & (fluid[2] < 0))
    slot = np.full(fluid[0].shape, -1, np.int32)
    slot[wet] = np.arange(int(wet.sum()), dtype=np.int32)
    slots = [slot] + [np.where(v[0] >= 0, v[0], -1).astype(np.int32) for v in vel]
    return solid, fluid, tuple(vel), slots, dense


def _csr_inputs(case, seed):
    """The pressure matrix of a liquid as the linear-solver module gets it."""
    sc = _csr_scene(case, seed)
    op = _operator(sc, sc.vel)
    on = op["unknown"]
    n = int(on.sum())
    num = torch.full(on.shape, -1, dtype=torch.int64, device=DEV)
    num[on] = torch.arange(n, device=DEV)
    rows, cols, vals = [num[on]], [num[on]], [op["diag"][on]]
    for d, c in enumerate(op["c"]):
        m = c != 0
        a, b = num[m], num[_shift(m, d)]
        rows += [a, b]
        cols += [b, a]
        vals += [-c[m], -c[m]]
    rows, cols, vals = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    order = torch.argsort(rows * n + cols)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return tuple(t.cpu().numpy() for t in (indptr, cols[order], vals[order], op["b"][on]))


def _shift(m, d):
    """The cells one further along axis d than those that m marks."""
    return torch.roll(m, 1, 2 - d)


# --------------------------------------------------------------------------
# the work that a call cannot do without


def _cells_faces(nx, ny, nz, dim):
    cells = nx * ny * nz
    faces = (nx + 1) * ny * nz + nx * (ny + 1) * nz + (nx * ny * (nz + 1) if dim == 3 else 0)
    nodes = (nx + 1) * (ny + 1) * (nz + 1 if dim == 3 else 1)
    return cells, faces, nodes


def _project_work(nx, ny, nz, dim):
    """The level sets and velocities read once, velocities and pressure written
    once; the arithmetic of one assembly, one residual and one update."""
    cells, faces, nodes = _cells_faces(nx, ny, nz, dim)
    return {"bytes": 4.0 * (nodes + cells + faces) + 4.0 * (faces + cells), "flops": 60.0 * cells}


def work(case):
    kind = case["kind"]
    if kind in ("project", "bricks"):
        return _project_work(case["nx"], case["ny"], case["nz"], case["dim"])
    if kind in ("batch", "served"):
        sizes, total = random.Random(int(case["mix"])), {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["count"]):
            e = _log_int(sizes, case["lo"], case["hi"])
            sizes.random()  # the scene's kind or pool
            w = _project_work(e, e, e, 3)
            for k in total:
                total[k] += w[k] * (1 if kind == "batch" else 3)
        return total
    if kind == "csr":
        cells = case["nx"] * case["ny"] * case["nz"]
        n = 0.37 * cells  # the liquid's share
        return {"bytes": n * (8 + 8 + 8 + 7 * 16), "flops": 14.0 * n}
    cells, faces, nodes = _cells_faces(case["nx"], case["ny"], case["nz"], case.get("dim", 3))
    if kind == "advect":
        # two traces per face and cell, each with an interpolation
        return {"bytes": 8.0 * (faces + cells) + 4.0 * cells, "flops": 100.0 * (faces + cells)}
    return {"bytes": 10.0 * faces + 4.0 * nodes, "flops": 10.0 * faces}


# --------------------------------------------------------------------------
# the same results in 64 bits


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        sc = _of_case(case, seed)
        p, vel = _project64(sc, sc.vel)
        return {"pressure": None if case["scene"] == "smoke" else p, "velocity": vel}
    if kind == "bricks":
        sc = _of_case(case, seed)
        slots, dense = _bricks_of(sc)[3:]
        p, vel = _project64(sc, dense)
        return [[None if a is p and case["scene"] == "smoke" else _gather_bricks(a, s), None]
                for a, s in zip([p] + vel, slots)]
    if kind in ("batch", "served"):
        scs = _mixed_scenes(case, seed)
        noise = _tick_noise(scs, seed) if kind == "served" else None
        ps, vels = [], []
        for n, sc in enumerate(scs):
            vel = sc.vel
            for tick in range(1 if kind == "batch" else 3):
                if tick:
                    vel = [v + t for v, t in zip(vel, noise[n][tick - 1])]
                p, vel = _project64(sc, vel)
            ps.append(p)
            vels.append(vel)
        smoke = any(sc.smoke for sc in scs)  # a smoke's pressure is defined up to a constant
        return {"pressure": None if smoke else torch.cat([p.reshape(-1) for p in ps]),
                "velocity": [torch.cat([v[d].reshape(-1) for v in vels]) for d in range(3)]}
    if kind == "advect":
        return _advect64(*_advect_inputs(case, seed))
    if kind == "after":
        return _after64(*_after_inputs(case, seed), case["width"])
    sc = _csr_scene(case, seed)
    op = _operator(sc, sc.vel)
    return _solve(op)[op["unknown"]].cpu().numpy()


def _gather_bricks(a, slot):
    nz, ny, nx = a.shape
    a = torch.nn.functional.pad(a, (0, (-nx) % 8, 0, (-ny) % 8, 0, (-nz) % 8))
    bz, by, bx = (n // 8 for n in a.shape)
    v = a.reshape(bz, 8, by, 8, bx, 8).permute(0, 2, 4, 1, 3, 5).reshape(-1, 512)
    s = torch.from_numpy(slot.astype(np.int64)).to(DEV)
    out = torch.empty((int((s >= 0).sum()), 512), dtype=F64, device=DEV)
    out[s[s >= 0]] = v[s >= 0]
    return out.reshape(-1).cpu().numpy()


# ---- projection


def _fraction(a, b):
    """The share of a segment with end values a, b on which they are negative."""
    cut = -torch.minimum(a, b) / (a - b).abs().clamp(min=1e-300)
    whole = ((a < 0) | (b < 0)).to(F64)
    return torch.where(a * b < 0, cut, whole)


def _square_fraction(v0, v1, v2, v3):
    """Area of the negative part of a unit square: the polygon of its inside
    corners and edge crossings, in corner order (shoelace sum)."""
    v, cx, cy = (v0, v1, v2, v3), (0.0, 1.0, 1.0, 0.0), (0.0, 0.0, 1.0, 1.0)
    zero = torch.zeros_like(v0)
    have = torch.zeros_like(v0, dtype=torch.bool)
    fx, fy, lx, ly, total = zero, zero, zero, zero, zero

    def add(on, x, y):
        nonlocal have, fx, fy, lx, ly, total
        total = torch.where(on & have, total + lx * y - ly * x, total)
        fx, fy = torch.where(on & ~have, x, fx), torch.where(on & ~have, y, fy)
        lx, ly = torch.where(on, x, lx), torch.where(on, y, ly)
        have = have | on

    for n in range(4):
        m = (n + 1) % 4
        add(v[n] < 0, zero + cx[n], zero + cy[n])
        cross = v[n] * v[m] < 0
        t = v[n] / torch.where(cross, v[n] - v[m], zero + 1.0)
        add(cross, (1 - t) * cx[n] + t * cx[m], (1 - t) * cy[n] + t * cy[m])
    total = total + lx * fy - ly * fx
    return 0.5 * total


def _inner(a, d, lo):
    """Entries [1:] (lo) or [:-1] of a along axis d."""
    n = a.shape[2 - d]
    return a.narrow(2 - d, 1 if lo else 0, n - 1)


def _clamped(x):
    return torch.where((x > 0) & (x < EPS), torch.full_like(x, EPS), x)


def _face_fractions(sc):
    """Open area and liquid share of the inner faces of each component."""
    s, f = sc.solid.to(F64), sc.fluid.to(F64)
    area, rho = [], []
    for d in range(sc.dim):
        if sc.dim == 3:
            e = [a for a in range(3) if a != d]
            q = [[_inner(_inner(s, e[0], i), e[1], j) for j in (0, 1)] for i in (0, 1)]
            a = 1.0 - _square_fraction(q[0][0], q[1][0], q[1][1], q[0][1])
        else:
            a = 1.0 - _fraction(_inner(s, 1 - d, 0), _inner(s, 1 - d, 1))
        n = a.shape[2 - d]
        area.append(_clamped(a.narrow(2 - d, 1, n - 2)))
        rho.append(_clamped(_fraction(_inner(f, d, 1), _inner(f, d, 0))))
    return area, rho


def _operator(sc, vel):
    """The pressure system: diagonal, couplings of each cell's + faces, right side."""
    area, rho = _face_fractions(sc)
    wet = sc.fluid < 0
    cells = _shapes(sc)[1]
    diag = torch.zeros(cells, dtype=F64, device=DEV)
    b = torch.zeros(cells, dtype=F64, device=DEV)
    linked = torch.zeros(cells, dtype=torch.bool, device=DEV)
    c = []
    for d in range(sc.dim):
        open_ = (area[d] > 0) & (rho[d] > 0)
        w = torch.where(open_, DT * area[d] / (sc.dx * sc.dx * torch.where(open_, rho[d], 1.0)), 0.0)
        u = vel[d].to(F64)
        q = area[d] * u.narrow(2 - d, 1, u.shape[2 - d] - 2) / sc.dx
        lo, hi = torch.nn.functional.pad(w, _pad1(d, 1, 0)), torch.nn.functional.pad(w, _pad1(d, 0, 1))
        diag += lo + hi
        b += torch.nn.functional.pad(q, _pad1(d, 1, 0)) - torch.nn.functional.pad(q, _pad1(d, 0, 1))
        both = open_ & _inner(wet, d, 1) & _inner(wet, d, 0)
        linked |= torch.nn.functional.pad(both, _pad1(d, 1, 0)) | torch.nn.functional.pad(both, _pad1(d, 0, 1))
        c.append(torch.nn.functional.pad(torch.where(both, w, 0.0), _pad1(d, 0, 1)))
    unknown = wet & linked
    return {"diag": torch.where(unknown, diag, 0.0), "b": torch.where(unknown, b, 0.0), "c": c, "unknown": unknown,
            "area": area, "rho": rho}


def _apply(op, x):
    y = op["diag"] * x
    for d, c in enumerate(op["c"]):
        n = c.shape[2 - d] - 1
        w = c.narrow(2 - d, 0, n)
        y.narrow(2 - d, 0, n).addcmul_(w, x.narrow(2 - d, 1, n), value=-1.0)
        y.narrow(2 - d, 1, n).addcmul_(w, x.narrow(2 - d, 0, n), value=-1.0)
    return y


def _solve(op, tol=1e-11):
    """Conjugate gradients with the diagonal as preconditioner, in 64 bits."""
    inv = torch.where(op["unknown"], 1.0 / torch.where(op["unknown"], op["diag"], 1.0), 0.0)
    r, x = op["b"].clone(), torch.zeros_like(op["b"])
    p = inv * r
    rz, stop = torch.sum(r * p), tol * float(r.norm())
    for it in range(20000):
        q = _apply(op, p)
        alpha = rz / torch.sum(p * q)
        x.addcmul_(alpha, p)
        r.addcmul_(alpha, q, value=-1.0)
        if it % 50 == 49 and float(r.norm()) <= stop:
            break
        z = inv * r
        rz, old = torch.sum(r * z), rz
        p = z.addcmul_(rz / old, p)
    return x


def _project64(sc, vel):
    op = _operator(sc, vel)
    p = _solve(op)
    out = []
    for d in range(sc.dim):
        open_ = (op["area"][d] > 0) & (op["rho"][d] > 0)
        grad = (_inner(p, d, 1) - _inner(p, d, 0)) / (torch.where(open_, op["rho"][d], 1.0) * sc.dx)
        u = vel[d].to(F64)
        inner = torch.where(open_, u.narrow(2 - d, 1, u.shape[2 - d] - 2) - DT * grad, 0.0)
        out.append(torch.nn.functional.pad(inner, _pad1(d, 1, 1)))
    return p, out


# ---- advection


def _corners(shape, pos):
    """Clamped positions' cells, weights and flat indices of the corners; axes
    x, y(, z) of a (z, y, x) array."""
    n = [shape[2], shape[1], shape[0]][: len(pos)]
    base, w, stride, s = 0, [], [], 1
    for p, m in zip(pos, n):
        p = p.clamp(0.0, m - 1.0)
        i = p.clamp(max=m - 2.0).floor()
        w.append((i + 1 - p, p - i))
        base = base + i.to(torch.int64) * s
        stride.append(s)
        s *= m
    out = []
    for k in range(1 << len(pos)):
        c, o = 1.0, base
        for a in range(len(pos)):
            c = c * w[a][(k >> a) & 1]
            o = o + ((k >> a) & 1) * stride[a]
        out.append((o, c))
    return out


def _interp(a, corners):
    f = a.reshape(-1)
    v = 0.0
    for o, c in corners:
        v = v + f[o] * c
    return v


def _full_velocity(sc, vel, d):
    """All components at the faces of component d (d = None: at the cells)."""
    out = []
    for c in range(sc.dim):
        u = vel[c]
        if c != d:
            u = 0.5 * (_inner(u, c, 0) + _inner(u, c, 1))  # at the cells
            if d is not None:  # the clamped mean of the two cells at a face
                lo = torch.cat([u.narrow(2 - d, 0, 1), u], 2 - d)
                u = 0.5 * (lo + torch.cat([u, u.narrow(2 - d, u.shape[2 - d] - 1, 1)], 2 - d))
        out.append(u)
    return out


def _trace(shape, u, sign, dx, dim):
    idx = []
    for a in range(dim):
        n = shape[2 - a]
        i = torch.arange(n, dtype=F64, device=DEV)
        i = i.reshape([-1 if 2 - a == k else 1 for k in range(3)])
        idx.append((i - sign * DT * u[a] / dx).expand(shape))
    return idx


def _maccormack64(sc, a, u_fwd, u_bwd_of, offs, fluid, hi0):
    """One array carried: forward, backward from the forward values, limited correction."""
    pos = _trace(a.shape, u_fwd, 1.0, sc.dx, sc.dim)
    moving = sum((u != 0) for u in u_fwd) > 0
    corners = _corners(a.shape, pos)
    fwd = torch.where(moving, _interp(a, corners), a)
    f = a.reshape(-1)
    lo, hi = torch.full_like(a, math.inf), torch.full_like(a, hi0)
    for o, _ in corners:
        lo, hi = torch.minimum(lo, f[o]), torch.maximum(hi, f[o])
    del corners
    lo, hi = torch.where(moving, lo, a), torch.where(moving, hi, a)
    at = [p + o for p, o in zip(pos, offs)]
    band = _interp(fluid, _corners(fluid.shape, at)) > -sc.dx
    yield fwd
    back = _interp(fwd, _corners(a.shape, _trace(a.shape, u_bwd_of(), -1.0, sc.dx, sc.dim)))
    value = fwd + 0.5 * (a - back)
    yield torch.where(band, fwd, torch.minimum(torch.maximum(value, lo), hi))


def _advect64(sc, q):
    vel, q, fluid = [v.to(F64) for v in sc.vel], q.to(F64), sc.fluid.to(F64)
    uc = _full_velocity(sc, vel, None)
    scalar = list(_maccormack64(sc, q, uc, lambda: uc, (0.0, 0.0, 0.0), fluid, 0.0))[1]
    fwd, steps = [None] * sc.dim, []
    for d in range(sc.dim):
        offs = [0.0, 0.0, 0.0]
        offs[d] = -0.5
        g = _maccormack64(sc, vel[d], _full_velocity(sc, vel, d), lambda d=d: _full_velocity(sc, fwd, d), offs, fluid,
                          0.0)
        fwd[d] = next(g)
        steps.append(g)
    return {"scalar": scalar, "velocity": [next(g) for g in steps]}


# ---- the steps after a projection


def _after64(sc, masks, width):
    vel, on = [v.to(F64) for v in sc.vel], [m.bool() for m in masks]
    for d in range(3):
        for _ in range(width):
            total, count = 0.0, 0.0
            for a in range(3):
                for side in (0, 1):
                    total = total + _neighbour(torch.where(on[d], vel[d], 0.0), a, side)
                    count = count + _neighbour(on[d].to(F64), a, side)
            new = ~on[d] & (count > 0)
            vel[d] = torch.where(new, total / count.clamp(min=1.0), vel[d])
            on[d] = on[d] | new
    solid, out = sc.solid.to(F64), []
    for d in range(3):
        shape = vel[d].shape
        ip = [torch.arange(shape[2 - a], dtype=F64, device=DEV).reshape([-1 if 2 - a == k else 1 for k in range(3)])
              .expand(shape) for a in range(3)]
        pos = [ip[a] + (0.0 if a == d else 0.5) for a in range(3)]
        inside = _interp(solid, _corners(solid.shape, pos)) < 0
        grad = [g / sc.dx for g in _gradient(solid, pos)]
        at = [_interp(vel[c], _corners(vel[c].shape, [pos[a] - (0.0 if a == c else 0.5) for a in range(3)]))
              for c in range(3)]
        dot = sum(a * g for a, g in zip(at, grad))
        v = torch.where(inside & (dot < 0) & on[d], at[d] - grad[d] * dot, vel[d])
        n = (sc.nx, sc.ny, sc.nz)[d]
        v = torch.where(on[d] & (ip[d] == 0) & (v < 0), 0.0, v)
        out.append(torch.where(on[d] & (ip[d] == n) & (v > 0), 0.0, v))
    return {"velocity": out, "active": [None] * 3}


def _neighbour(a, axis, side):
    """a one cell further (side 0) or nearer along the axis, 0 beyond the ends."""
    n = a.shape[2 - axis] - 1
    return torch.nn.functional.pad(a.narrow(2 - axis, 1 - side, n), _pad1(axis, side, 1 - side))


def _gradient(a, pos):
    """Gradient of the trilinear interpolant, per cell."""
    n = [a.shape[2], a.shape[1], a.shape[0]]
    cell = [p.clamp(0.0, m - 1.0).clamp(max=m - 2.0).floor() for p, m in zip(pos, n)]
    out = []
    for d in range(3):
        lo = [c if k == d else p for k, (c, p) in enumerate(zip(cell, pos))]
        hi = [c + 1 if k == d else p for k, (c, p) in enumerate(zip(cell, pos))]
        out.append(_interp(a, _corners(a.shape, hi)) - _interp(a, _corners(a.shape, lo)))
    return out
