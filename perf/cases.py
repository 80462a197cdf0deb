"""Performance cases of the WCSPH step: what is timed, and what it should return.

A case is one piece of work as a user's program does it through the public
entry points: `FluidSystem` (set a state, advance, export frames), `Batch`
(many scenes per step, every scene read back) or `Server` (requests submitted
and fetched).  `listed()` names the cases, `draw(rng)` gives more of the same
ranges, `prepare` makes a case's inputs and handles from a seed, `run` is one
pass, `work` what a pass cannot do without, and `exact` the same outputs
computed in 64 bits by plain torch.

Fluid blocks are lattices with uniform jitter and a smooth initial motion of
up to 0.2 m/s, as a block that is already under way has it.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from libfluid_gb300 import FluidSystem
from libfluid_gb300.batch import Batch
from libfluid_gb300.server import Server
from libfluid_gb300.workloads import SceneSpec

# bytes a substep cannot do without, per particle (position, velocity and
# acceleration read and written) and per cell (count and start), the bytes of
# one exported frame, and the operations of one neighbour pair (density and
# XSPH about 25, pressure and viscosity about 50, normals and tension 40)
STATE_BYTES, CELL_BYTES, EXPORT_BYTES = 72, 8, 36
PAIR_FLOPS, TENSION_FLOPS = 75, 40


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _dam(name, nx, ny, nz, spacing, box, dt, frames, substeps, restart=True, **kw):
    c = dict(name=name, kind="frames", scene="dam", nx=nx, ny=ny, nz=nz, spacing=spacing, box_x=box[0],
             box_y=box[1], box_z=box[2], res=0, jitter=0.05, squeeze=1.0, tension=0.0, viscosity=0.01,
             adhesion=0.0, c0=20.0, dt=dt, frames=frames, substeps=substeps, restart=restart)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest use: a 12^3 block, four frames of one substep; launches and waits decide
        _dam("tiny_1728", 12, 12, 12, 0.01, (0.4, 0.3, 0.3), 2e-4, 4, 1),
        # the reference driver's defaults: two dam breaks of 5,000 particles in the unit cube, res 16, surface
        # tension and adhesion on, one substep per exported frame
        _dam("fluidtest_10k", 11, 29, 16, 0.0, (1.0, 1.0, 1.0), 2e-3, 8, 1, scene="double", res=16, tension=1.0,
             viscosity=0.2, adhesion=0.1, c0=10.0, particles=10000),
        # the small dam break, 32,768 particles: four frames of ten substeps
        _dam("small_dam_32k", 32, 32, 32, 0.01, (1.0, 0.6, 0.6), 2e-4, 4, 10),
        # the sphere boundary with surface tension: about 82,000 particles in a sphere
        _dam("sphere_tank_82k", 70, 70, 70, 0.01, (0.7, 0.7, 0.7), 2e-4, 2, 5, scene="sphere", tension=0.05),
        # an odd block with surface tension: sizes that fill no tile
        _dam("odd_tension_250k", 63, 61, 65, 0.005, (0.63, 0.41, 0.39), 1e-4, 1, 10, tension=0.0728),
        # the 1M dam break played frame by frame: every substep exported
        _dam("dam_1m_frames", 100, 100, 100, 0.005, (2.0, 1.0, 1.0), 1e-4, 8, 1),
        # the 1M dam break simulated: twenty substeps, then an export
        _dam("dam_1m", 100, 100, 100, 0.005, (2.0, 1.0, 1.0), 1e-4, 1, 20),
        # the same block late in a run, in the unit cube: no lattice left, the bottom squeezed (a third more
        # neighbours, cell rows past 32 candidates), particles changing cells in every substep
        _dam("late_1m", 100, 100, 100, 0.005, (1.0, 1.0, 1.0), 1e-4, 1, 2, restart=False, res=100, jitter=0.3,
             squeeze=0.7),
        # about 8M particles with surface tension, a pool and two falling spheres: the largest
        _dam("pool_8m", 200, 180, 200, 0.005, (1.0, 2.0, 1.0), 8e-5, 1, 2, restart=False, scene="pool",
             tension=0.0728, c0=25.0),
        # 256 scenes of 2,048 to 65,536 particles advanced together, every scene read back
        dict(name="batch_256", kind="batch", scenes=256, nmin=2048, nmax=65536, substeps=20),
        # requests of 1,024 to 131,072 particles and 10 to 40 substeps, served by continuous batching
        dict(name="served_32", kind="served", requests=32, nmin=1024, nmax=131072, steps_min=10, steps_max=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dam", "dam", "dam", "late", "late", "double", "sphere", "batch", "served"])
    if kind == "batch":
        nmin = _log(rng, 1024, 4096)
        return dict(kind="batch", scenes=_log(rng, 16, 200), nmin=nmin, nmax=_log(rng, 2 * nmin, 65536),
                    substeps=rng.randint(5, 20))
    if kind == "served":
        return dict(kind="served", requests=_log(rng, 8, 32), nmin=1024, nmax=_log(rng, 4096, 131072),
                    steps_min=rng.randint(5, 10), steps_max=rng.randint(15, 40))
    tension = rng.choice([0.0, 0.0, round(rng.uniform(0.01, 0.0728), 4)])
    visc = round(rng.uniform(0.005, 0.05), 4)
    if kind == "sphere":
        m = rng.randint(20, 90)
        c = _dam("", m, m, m, 0.01, (m * 0.01,) * 3, 2e-4, rng.randint(1, 3), rng.randint(1, 5), scene="sphere",
                 tension=tension, viscosity=visc)
    elif kind == "double":
        n, res = _log(rng, 2000, 60000), rng.randint(12, 24)
        c = _dam("", 1, 1, 1, 0.0, (1.0, 1.0, 1.0), 2e-3, rng.randint(2, 8), 1, scene="double", res=res,
                 particles=n, tension=rng.choice([0.0, 1.0]), viscosity=0.2, adhesion=0.1, c0=10.0)
    else:
        n = _log(rng, 1000, 2_000_000 if kind == "dam" else 1_000_000)
        ay, az = rng.uniform(0.5, 2.0), rng.uniform(0.5, 2.0)
        nx = max(6, round((n / (ay * az)) ** (1 / 3)))
        ny, nz = max(6, round(nx * ay)), max(6, round(nx * az))
        s = 0.01 if n < 200_000 else 0.005
        dt = 2e-4 if n < 200_000 else 1e-4
        box = tuple(round(f * k * s, 4) for f, k in ((rng.uniform(1.2, 3), nx), (rng.uniform(1.1, 2), ny),
                                                     (rng.uniform(1.1, 2), nz)))
        if kind == "late":
            c = _dam("", nx, ny, nz, s, box, dt, 1, 2, restart=n < 50_000, jitter=round(rng.uniform(0.15, 0.35), 3),
                     squeeze=round(rng.uniform(0.6, 0.95), 3), tension=tension, viscosity=visc)
        else:
            c = _dam("", nx, ny, nz, s, box, dt, rng.randint(1, 4), rng.choice([1, 2, 5, 10]), tension=tension,
                     viscosity=visc)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _lattice(nx, ny, nz, s):
    g = np.meshgrid(*[(np.arange(k, dtype=np.float32) + np.float32(0.5)) * np.float32(s) for k in (nx, ny, nz)],
                    indexing="ij", copy=False)
    return np.stack([a.reshape(-1) for a in g], 1)


def _ball(center, radius, s):
    lo = [int(math.floor((c - radius) / s)) for c in center]
    k = [int(math.ceil((c + radius) / s)) - a for c, a in zip(center, lo)]
    p = _lattice(*k, s) + np.asarray(lo, np.float32) * np.float32(s)
    return p[((p - np.asarray(center, np.float32)) ** 2).sum(1) <= radius * radius]


def _motion(pos, box, rng):
    """A smooth motion of up to 0.2 m/s whose component towards each wall is not zero there."""
    ph = rng.uniform(0.6, 1.4, 3).astype(np.float32)
    x = pos / np.asarray(box, np.float32)
    v = np.empty_like(pos)
    for a in range(3):
        b = (a + 1) % 3
        v[:, a] = np.float32(0.12) * np.cos(np.float32(3.0) * x[:, a] + ph[a]) + \
            np.float32(0.06) * np.sin(np.float32(5.0) * x[:, b] + ph[b])
    return v


def _scene(case, seed):
    """(parameters, positions, velocities) of a `frames` case."""
    rng = np.random.default_rng([int(seed), 1])
    s, box = case["spacing"], (case["box_x"], case["box_y"], case["box_z"])
    h = 1.0 / case["res"] if case["res"] else 2.0 * s
    mass, psize, fall = 1000.0 * s ** 3, 0.5 * s, None
    if case["scene"] == "double":
        # two columns in opposite corners, as the reference driver builds them
        half = case["particles"] // 2
        vol = 0.33 * 0.9 * 0.33 / half
        s = vol ** (1 / 3)
        k = [int(0.33 / s), 1 + int(0.9 / s), 1 + int(0.33 / s)]
        one = _lattice(*k, s)
        one = one[(one < np.asarray((0.33, 0.9, 0.33), np.float32)).all(1)][:half]
        pos = np.concatenate([one, one + np.asarray((0.66, 0.0, 0.66), np.float32)])
        mass, psize = vol * 1000.0, 0.5 * s
    elif case["scene"] == "sphere":
        r = 0.5 * case["nx"] * s
        pos = _ball((r, r, r), r - s, s)
        pos = pos[pos[:, 1] <= r]
    elif case["scene"] == "pool":
        pool = _lattice(case["nx"], case["ny"], case["nz"], s)
        balls = [_ball(c, 0.229, s) for c in ((0.27, 1.3, 0.5), (0.73, 1.6, 0.5))]
        fall = pool.shape[0]
        pos = np.concatenate([pool] + balls)
    else:
        pos = _lattice(case["nx"], case["ny"], case["nz"], s)
    if case["squeeze"] < 1.0:
        # spacing `squeeze` at the bottom, 1 at the top
        top = case["ny"] * s
        y = pos[:, 1] / np.float32(top)
        pos[:, 1] = np.float32(top) * y * (np.float32(case["squeeze"]) + np.float32(1.0 - case["squeeze"]) * y)
    pos += (rng.random(pos.shape, dtype=np.float32) * np.float32(2) - np.float32(1)) * np.float32(case["jitter"] * s)
    if case["scene"] != "sphere":
        edge = np.float32(0.1 * s)
        np.clip(pos, edge, np.asarray(box, np.float32) - edge, out=pos)
    vel = _motion(pos, box, rng)
    if fall is not None:
        vel[fall:] = np.asarray((0.0, -1.0, 0.0), np.float32)
    prm = dict(box=box, res=case["res"], h=h, rest_density=1000.0, mass=mass, particle_size=psize, gamma=7.0,
               gas_constant=case["c0"] ** 2, viscosity=case["viscosity"], xsph=0.5, surface_tension=case["tension"],
               adhesion=case["adhesion"], vdamp=0.5, vel_limit=5.0, acc_limit=150.0, gravity=(0.0, -9.81, 0.0),
               dt=_part_dt(case), boundary=1 if case["scene"] == "sphere" else 0)
    return prm, pos, vel


def _mixed_sizes(case, count):
    """Block sizes of a batch or of a request set: the case's, whatever the seed."""
    r = random.Random(count * 1000003 + case["nmin"] * 31 + case["nmax"])
    out = []
    for _ in range(count):
        n = math.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        ay, az = r.uniform(0.5, 2.0), r.uniform(0.5, 2.0)
        nx = max(2, round((n / (ay * az)) ** (1 / 3)))
        out.append((nx, max(2, round(nx * ay)), max(2, round(nx * az)), r.uniform(0.005, 0.05), r.uniform(0.0, 0.07)))
    return out


def _mixed_scenes(case, seed, count):
    """Dam breaks of mixed sizes: [(parameters, positions, velocities)]."""
    s = 0.01
    out = []
    for k, (nx, ny, nz, visc, tension) in enumerate(_mixed_sizes(case, count)):
        rng = np.random.default_rng([int(seed), 2, k])
        box = (2.0 * nx * s, 1.2 * ny * s, 1.2 * nz * s)
        pos = _lattice(nx, ny, nz, s)
        pos += (rng.random(pos.shape, dtype=np.float32) * np.float32(2) - np.float32(1)) * np.float32(0.05 * s)
        prm = dict(box=box, res=0, h=2.0 * s, rest_density=1000.0, mass=1000.0 * s ** 3, particle_size=0.5 * s,
                   gamma=7.0, gas_constant=400.0, viscosity=visc, xsph=0.5, surface_tension=tension, adhesion=0.0,
                   vdamp=0.5, vel_limit=5.0, acc_limit=150.0, gravity=(0.0, -9.81, 0.0), dt=2e-4, boundary=0)
        out.append((prm, pos, _motion(pos, box, rng)))
    return out


def _request_steps(case):
    r = random.Random(case["requests"] * 7919 + case["steps_max"])
    return [r.randint(case["steps_min"], case["steps_max"]) for _ in range(case["requests"])]


def _part_dt(case):
    return float(np.float32(case["dt"] * case["substeps"]) / np.float32(case["substeps"]))


def _substeps(case):
    """Substeps one advance(dt * substeps, substeps) runs: the reference's float loop."""
    full = np.float32(case["dt"] * case["substeps"])
    part = full / np.float32(case["substeps"])
    t, k = part, 0
    while t <= full:
        k, t = k + 1, np.float32(t + part)
    return k


def _spec(prm, pos, vel):
    return SceneSpec(box=prm["box"], h=prm["h"], blocks=[], rest_density=prm["rest_density"], mass=prm["mass"],
                     gamma=prm["gamma"], gas_constant=prm["gas_constant"], viscosity=prm["viscosity"],
                     xsph=prm["xsph"], surface_tension=prm["surface_tension"], adhesion=prm["adhesion"],
                     vdamp=prm["vdamp"], particle_size=prm["particle_size"], vel_limit=prm["vel_limit"],
                     acc_limit=prm["acc_limit"], gravity=prm["gravity"], dt=prm["dt"], extra_pos=pos, extra_vel=vel)


def prepare(case, seed):
    if case["kind"] == "batch":
        b = Batch()
        ids = [b.add_scene(_spec(*sc)) for sc in _mixed_scenes(case, seed, case["scenes"])]
        return dict(kind="batch", batch=b, ids=ids, substeps=case["substeps"])
    if case["kind"] == "served":
        reqs = [(_spec(*sc), k, sc[1], sc[2])
                for sc, k in zip(_mixed_scenes(case, seed, case["requests"]), _request_steps(case))]
        return dict(kind="served", server=Server(memory_budget=100 << 30), requests=reqs)
    prm, pos, vel = _scene(case, seed)
    fs = FluidSystem()
    fs.init(pos.shape[0], case["res"] or 1)
    if not case["res"]:
        fs.setDomain(*prm["box"], prm["h"])
    if prm["boundary"]:
        fs.setBoundary(prm["boundary"])
    fs.setParams(**{k: prm[k] for k in ("rest_density", "mass", "gamma", "gas_constant", "viscosity", "xsph",
                                        "surface_tension", "adhesion", "vdamp", "particle_size", "vel_limit",
                                        "acc_limit", "gravity", "dt")})
    fs.setState(pos, vel)
    return dict(kind="frames", fs=fs, pos=pos, vel=vel, out=[np.zeros_like(pos) for _ in range(3)],
                frames=case["frames"], substeps=case["substeps"], frame_dt=case["dt"] * case["substeps"],
                restart=case["restart"])


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    if state["kind"] == "frames":
        # a clip from a given state (or, without restart, the next frames of a running one)
        fs = state["fs"]
        if state["restart"]:
            fs.setState(state["pos"], state["vel"])
        for _ in range(state["frames"]):
            fs.advance(state["frame_dt"], state["substeps"])
            fs.exportToData(*state["out"])
        return dict(zip(("points", "colour", "velocity"), state["out"]))
    if state["kind"] == "batch":
        b = state["batch"]
        b.step(state["substeps"])
        got = [b.get_state(i) for i in state["ids"]]
    else:
        sv = state["server"]
        rids = [sv.submit(spec, k, pos=pos, vel=vel) for spec, k, pos, vel in state["requests"]]
        sv.drain()
        got = [sv.fetch(r) for r in rids]
    return {k: np.concatenate([g[q] for g in got])
            for q, k in enumerate(("points", "colour", "velocity") if len(got[0]) == 3 else ("points", "velocity"))}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _cells(prm):
    if prm["res"]:
        return prm["res"] ** 3
    return int(np.prod([max(1, math.ceil(l / prm["h"] - 1e-3)) for l in prm["box"]]))


def work(case):
    if case["kind"] == "frames":
        prm, pos, _ = _scene(case, 0)
        k = case["frames"] * _substeps(case)
        sets = [(pos.shape[0], _cells(prm), k, prm["surface_tension"], prm["h"], prm["mass"])]
        io = EXPORT_BYTES * case["frames"] * pos.shape[0] + (24 * pos.shape[0] if case["restart"] else 0)
    else:
        count = case["scenes"] if case["kind"] == "batch" else case["requests"]
        steps = [case["substeps"]] * count if case["kind"] == "batch" else _request_steps(case)
        sets = []
        for (nx, ny, nz, _, tension), k in zip(_mixed_sizes(case, count), steps):
            cells = _cells(dict(res=0, h=0.02, box=(0.02 * nx, 0.012 * ny, 0.012 * nz)))
            sets.append((nx * ny * nz, cells, k, tension, 0.02, 1e-3))
        io = sum(x[0] for x in sets) * (EXPORT_BYTES if case["kind"] == "batch" else 48)
    byte, flop = io, 0
    for n, cells, k, tension, h, mass in sets:
        nbr = 4.0 / 3.0 * math.pi * h ** 3 * 1000.0 / mass
        byte += k * (n * STATE_BYTES + cells * CELL_BYTES)
        flop += k * n * nbr * (PAIR_FLOPS + (TENSION_FLOPS if tension else 0))
    return {"bytes": byte, "flops": flop}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
_PRM = ("h", "rest_density", "mass", "particle_size", "gamma", "gas_constant", "viscosity", "xsph",
        "surface_tension", "adhesion", "vdamp", "vel_limit", "acc_limit", "dt")
_CHUNK = 400_000
_TINY = 1.1754943508222875e-38


def _tables(prms, dev):
    """Per-scene parameters in 64 bits of the FP32 values a caller passes."""
    t = {k: torch.tensor([float(np.float32(p[k])) for p in prms], dtype=torch.float64, device=dev) for k in _PRM}
    t["g"] = torch.tensor([[float(np.float32(x)) for x in p["gravity"]] for p in prms], dtype=torch.float64,
                          device=dev)
    box, dims, inv = [], [], []
    for p in prms:
        if p["res"]:
            box.append([1.0] * 3)
            dims.append([p["res"]] * 3)
            inv.append(float(p["res"]))
        else:
            h = np.float32(p["h"])
            box.append([float(np.float32(x)) for x in p["box"]])
            dims.append([max(1, math.ceil(x / float(h) - 1e-3)) for x in box[-1]])
            inv.append(float(np.float32(1.0) / h))
    t["half"] = 0.5 * torch.tensor(box, dtype=torch.float64, device=dev)
    t["dims"] = torch.tensor(dims, dtype=torch.int64, device=dev)
    t["inv"] = torch.tensor(inv, dtype=torch.float32, device=dev)
    cells = t["dims"].prod(1)
    t["base"] = torch.cumsum(cells, 0) - cells
    t["cells"] = int(cells.sum())
    t["sphere"] = torch.tensor([bool(p["boundary"]) for p in prms], device=dev)
    h = t["h"]
    t["poly6"] = 315.0 / (64.0 * math.pi * h ** 9)
    t["grad_poly6"] = -945.0 / (32.0 * math.pi * h ** 9)
    t["grad_spiky"] = -45.0 / (math.pi * h ** 6)
    t["eos"] = t["gas_constant"] * t["rest_density"] / t["gamma"]
    return t


def _sdf(t, sc, p):
    half = t["half"][sc]
    q = (p - half).abs() - half
    box = q.max(1).values.clamp(max=0.0) + q.clamp(min=0.0).norm(dim=1)
    ball = (p - half).norm(dim=1) - half.min(1).values
    return torch.where(t["sphere"][sc], ball, box)


def _sdf_normal(t, sc, p):
    e = 0.0001
    n = []
    for a in range(3):
        d = torch.zeros(3, dtype=p.dtype, device=p.device)
        d[a] = e
        n.append(_sdf(t, sc, p + d) - _sdf(t, sc, p - d))
    n = torch.stack(n, 1)
    return n / n.norm(dim=1, keepdim=True)


def _pairs(t, sc, cell, start, pos, h2):
    """Chunks (i, j) of the pairs within h at `pos` whose cells are neighbours."""
    n = pos.shape[0]
    dims = t["dims"][sc]
    for lo in range(0, n, _CHUNK):
        hi = min(n, lo + _CHUNK)
        ii, jj = [], []
        c, d, b = cell[lo:hi], dims[lo:hi], t["base"][sc[lo:hi]]
        x0, x1 = (c[:, 0] - 1).clamp(min=0), torch.minimum(c[:, 0] + 1, d[:, 0] - 1)
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                y, z = c[:, 1] + dy, c[:, 2] + dz
                ok = (y >= 0) & (y < d[:, 1]) & (z >= 0) & (z < d[:, 2])
                row = b + torch.where(ok, y * d[:, 0] + z * d[:, 0] * d[:, 1], torch.zeros_like(y))
                j0 = start[row + x0]
                cnt = torch.where(ok, start[row + x1 + 1] - j0, torch.zeros_like(j0))
                i = torch.repeat_interleave(torch.arange(hi - lo, device=pos.device), cnt)
                j = torch.arange(i.numel(), device=pos.device) - (torch.cumsum(cnt, 0) - cnt)[i] + j0[i]
                i = i + lo
                r = pos[i] - pos[j]
                m = ((r * r).sum(1) <= h2[i]) & (i != j)
                ii.append(i[m])
                jj.append(j[m])
        yield torch.cat(ii), torch.cat(jj)


def _step64(t, sc, p, p32, v, a):
    """One substep; returns the state in cell order, its densities, and that order.

    `p32` follows the positions with the storage rounding of FP32: the cell
    of a particle, and with it the order of the outputs, is defined on those."""
    g = {k: t[k][sc] for k in _PRM + ("poly6", "grad_poly6", "grad_spiky", "eos")}
    grav = t["g"][sc]
    h, h2, mass = g["h"], g["h"] ** 2, g["mass"]
    # the sort
    cell = torch.floor(p32 * t["inv"][sc][:, None]).to(torch.int64)
    dims = t["dims"][sc]
    key = t["base"][sc] + cell[:, 0] + cell[:, 1] * dims[:, 0] + cell[:, 2] * dims[:, 0] * dims[:, 1]
    order = torch.argsort(key, stable=True)
    # scenes are contiguous in the key, so the per-particle tables stay valid
    p, p32, v, a, cell = p[order], p32[order], v[order], a[order], cell[order]
    count = torch.bincount(key, minlength=t["cells"])
    start = torch.cat([torch.zeros(1, dtype=torch.int64, device=p.device), torch.cumsum(count, 0)])
    # density and pressure
    total = torch.zeros_like(h)
    pairs = []
    for i, j in _pairs(t, sc, cell, start, p, h2):
        x = (h2[i] - ((p[i] - p[j]) ** 2).sum(1)).clamp(min=0.0)
        total.index_add_(0, i, mass[i] * g["poly6"][i] * x ** 3)
        pairs.append((i.to(torch.int32), j.to(torch.int32)))
    d = _sdf(t, sc, p).abs()
    c = -d
    poly = c ** 3 * (35 * c ** 6 - 180 * c ** 4 * h2 + 378 * c ** 2 * h ** 4 - 420 * h ** 6) + \
        315 * c * h ** 8 + 128 * h ** 9
    wall = torch.where(d < h, g["rest_density"] * (0.0039062 / h ** 9) * poly, torch.zeros_like(h))
    corr = total + wall
    rho = torch.where(total == 0, g["rest_density"], corr)
    ratio = corr / g["rest_density"]
    prs = torch.where(corr == 0, torch.zeros_like(h), g["eos"] * (ratio ** g["gamma"] - 1))
    cs = g["gas_constant"] * ratio ** (g["gamma"] - 1)
    tension = bool((g["surface_tension"] != 0).any())
    nrm = torch.zeros_like(p)
    if tension:
        for i, j in pairs:
            i, j = i.long(), j.long()
            r = p[i] - p[j]
            r2 = (r * r).sum(1)
            w = mass[i] * g["grad_poly6"][i] * (h2[i] - r2).clamp(min=0.0) ** 2 / rho[j]
            ok = (r2 > _TINY) & (rho[j] > _TINY)
            nrm.index_add_(0, i, torch.where(ok, w, torch.zeros_like(w))[:, None] * r)
        nrm = nrm * h[:, None]
    # forces
    fp, fv, ft = torch.zeros_like(p), torch.zeros_like(p), torch.zeros_like(p)
    for i, j in pairs:
        i, j = i.long(), j.long()
        r = p[j] - p[i]
        r2 = (r * r).sum(1)
        ok = (r2 > _TINY) & (rho[j] > _TINY)
        i, j, r, r2 = i[ok], j[ok], r[ok], r2[ok]
        rl, hi = r2.sqrt(), h[i]
        ux = -((v[i] - v[j]) * r).sum(1)
        visc = torch.where(ux < 0, -g["viscosity"][i] * (cs[i] + cs[j]) * hi * ux /
                           ((r2 + 0.01 * hi * hi) * (rho[i] + rho[j])), torch.zeros_like(ux))
        mid = prs[j] / rho[i] ** 2 + prs[i] / rho[j] ** 2
        grad = (mass[i] * g["grad_spiky"][i] * (hi - rl).clamp(min=0.0) ** 2 / rl)[:, None] * r
        fp.index_add_(0, i, grad * mid[:, None])
        fv.index_add_(0, i, grad * (mid + visc)[:, None])
        if tension:
            near = (hi - rl) ** 3 * rl ** 3
            coh = torch.where(rl > 0.5 * hi, near, 2 * near - hi ** 6 * 0.0156)
            coh = torch.where(rl >= hi, torch.zeros_like(coh), coh)
            both = (-mass[i] ** 2 * coh / rl)[:, None] * r - \
                (g["surface_tension"][i] * mass[i])[:, None] * (nrm[i] - nrm[j])
            ft.index_add_(0, i, (g["rest_density"][i] / rho[i])[:, None] * both)
    fv, ft = fv * g["viscosity"][:, None], ft * g["surface_tension"][:, None]
    z = -_sdf(t, sc, p).clamp(max=0.0) * 0.25 / g["particle_size"]
    sticky = (z < 1) & (g["adhesion"] != 0)
    fa = torch.zeros_like(p)
    if bool(sticky.any()):
        k = sticky.nonzero()[:, 0]
        s = g["adhesion"][k] * rho[k] / g["rest_density"][k] / (1 - z[k]) ** 3
        fa[k] = s[:, None] * _sdf_normal(t, sc[k], p[k])
    del pairs
    # integrator and boundary
    an = (fp + ft + fv + fa) * mass[:, None] + grav
    al = an.norm(dim=1)
    an = an * torch.where(al > g["acc_limit"], g["acc_limit"] / al, torch.ones_like(al))[:, None]
    dt = g["dt"][:, None]
    pn = p + v * dt + 0.5 * a * dt * dt
    move = (v * dt + (0.5 * a * dt * dt).float().double()).float()
    pn32 = p32 + move
    vn = v + 0.5 * (a + an) * dt
    vl = vn.norm(dim=1)
    vn = vn * torch.where(vl > g["vel_limit"], g["vel_limit"] / vl, torch.ones_like(vl))[:, None]
    d = _sdf(t, sc, pn)
    k = (d > -g["particle_size"]).nonzero()[:, 0]
    if k.numel():
        nb = _sdf_normal(t, sc[k], pn[k])
        s = -(d[k] + g["particle_size"][k])[:, None] * nb
        pn[k] += s
        pn32[k] = (pn32[k].double() + s).float()
        vn[k] -= ((1 + g["vdamp"][k]) * (nb * vn[k]).sum(1))[:, None] * nb
    # XSPH over this substep's cell lists at the new positions
    dv = torch.zeros_like(vn)
    for i, j in _pairs(t, sc, cell, start, pn, h2):
        x = (h2[i] - ((pn[i] - pn[j]) ** 2).sum(1)).clamp(min=0.0)
        rs = rho[i] + rho[j]
        w = torch.where(rs > _TINY, g["poly6"][i] * x ** 3 * 2 * mass[i] / rs, torch.zeros_like(x))
        dv.index_add_(0, i, w[:, None] * (vn[j] - vn[i]))
    return pn, pn32, vn + g["xsph"][:, None] * dv, an, rho, order


def _colour(ratio):
    r, gr, b = torch.ones_like(ratio), torch.zeros_like(ratio), torch.zeros_like(ratio)
    lo, mid = ratio < 1, (ratio >= 1) & (ratio < 2)
    r[lo], gr[lo], b[lo] = 0.0, ratio[lo], 1 - ratio[lo]
    r[mid], gr[mid] = ratio[mid] - 1, 2 - ratio[mid]
    return torch.stack([r, gr, b], 1)


def _simulate64(scenes, steps):
    """Final (points, colour, velocity) of each scene after its substeps."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = [None] * len(scenes)
    ids = list(range(len(scenes)))
    p32 = [torch.from_numpy(s[1]).to(dev) for s in scenes]
    v = [torch.from_numpy(s[2]).to(dev).double() for s in scenes]
    p = [x.double() for x in p32]
    a = [torch.zeros_like(x) for x in p]
    done = 0
    while ids:
        k = min(steps[s] for s in ids) - done
        t = _tables([scenes[s][0] for s in ids], dev)
        ns = [scenes[s][1].shape[0] for s in ids]
        sc = torch.repeat_interleave(torch.arange(len(ids), device=dev), torch.tensor(ns, device=dev))
        cp, c32, cv, ca = (torch.cat([x[s] for s in ids]) for x in (p, p32, v, a))
        rho = None
        for _ in range(k):
            cp, c32, cv, ca, rho, _ = _step64(t, sc, cp, c32, cv, ca)
        done += k
        for s, *x in zip(ids, *(y.split(ns) for y in (cp, c32, cv, ca, rho))):
            p[s], p32[s], v[s], a[s] = x[:4]
            if steps[s] == done:
                out[s] = (x[0], _colour(x[4] / float(np.float32(scenes[s][0]["rest_density"]))), x[2])
        ids = [s for s in ids if steps[s] > done]
    return out


def exact(case, seed):
    if case["kind"] == "frames":
        scenes, steps = [_scene(case, seed)], [case["frames"] * _substeps(case)]
    elif case["kind"] == "batch":
        scenes = _mixed_scenes(case, seed, case["scenes"])
        steps = [case["substeps"]] * len(scenes)
    else:
        scenes, steps = _mixed_scenes(case, seed, case["requests"]), _request_steps(case)
    got = _simulate64(scenes, steps)
    keys = ("points", "velocity") if case["kind"] == "served" else ("points", "colour", "velocity")
    at = {"points": 0, "colour": 1, "velocity": 2}
    return {k: torch.cat([x[at[k]] for x in got]) for k in keys}
