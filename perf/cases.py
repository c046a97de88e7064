"""Performance cases of the grid-step path, each a call sequence that a scene
script makes: advection, pressure solves, whole smoke steps, the FLIP
transfers, velocity and levelset extrapolation, and a batch of small scenes.

Inputs come from a seed alone (smooth random flows, plume-shaped densities,
dam-break surfaces, jittered particles) and reach the GPU through the same
array uploads that a script uses.  Outputs are the grids' device storage.
"""
import ctypes
import math

import numpy as np
import torch

import mantaflow_gb300 as m
from mantaflow_gb300 import _lib
from mantaflow_gb300 import batch as mb

FLUID, OBSTACLE, EMPTY, OUTFLOW = m.FlagFluid, m.FlagObstacle, m.FlagEmpty, m.FlagOutflow
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ----------------------------------------------------------------- the cases
def listed():
    return [
        # a small scene's smoke density, once per step: launches and latency count
        {"name": "advect_density_73x66x57", "kind": "advect", "grid": "density", "order": 2, "nx": 73, "ny": 66, "nz": 57},
        # the largest self-advection of a production-size velocity field
        {"name": "advect_velocity_256", "kind": "advect", "grid": "velocity", "order": 2, "nx": 256, "ny": 256, "nz": 256},
        # a liquid scene's surface, first order as the free-surface scenes take it, rows of an odd length
        {"name": "advect_levelset_129x97x128", "kind": "advect", "grid": "levelset", "order": 1, "nx": 129, "ny": 97, "nz": 128},
        # the default solver (MIC(0)) at the size of the smoke examples
        {"name": "solve_smoke_mic_64", "kind": "solve", "scene": "smoke", "pc": "mic", "nx": 64, "ny": 64, "nz": 64},
        # the default solver on a dam break with ghost-fluid surfaces
        {"name": "solve_liquid_mic_128", "kind": "solve", "scene": "liquid", "pc": "mic", "nx": 128, "ny": 128, "nz": 128},
        # the static multigrid solver around an obstacle, sizes that divide by nothing
        {"name": "solve_obstacle_mg_161x199x143", "kind": "solve", "scene": "obstacle", "pc": "mgstatic", "nx": 161, "ny": 199, "nz": 143},
        # a whole smoke step, large, with the solver such scenes use
        {"name": "step_smoke_mg_256", "kind": "step", "pc": "mgstatic", "nx": 256, "ny": 256, "nz": 256},
        # a whole smoke step in 2D, the size of an interactive preview
        {"name": "step_smoke2d_96x128", "kind": "step", "pc": "mic", "nx": 96, "ny": 128, "nz": 1},
        # particles to grid, a full tank in seeding order with eight particles per cell
        {"name": "flip_splat_128", "kind": "flip_splat", "fill": "tank", "ppc": 8, "shuffled": False, "nx": 128, "ny": 128, "nz": 128},
        # the transfers of one FLIP step on a dam whose particles have been mixed by the flow
        {"name": "flip_cycle_75x62x90", "kind": "flip_cycle", "fill": "dam", "ppc": 8, "shuffled": True, "nx": 75, "ny": 62, "nz": 90},
        # velocities and levelset carried out of the liquid before advection
        {"name": "extrapolate_128", "kind": "extrapolate", "distance": 4, "nx": 128, "ny": 128, "nz": 128},
        # many small smoke scenes at once (training data), four steps per saved frame
        {"name": "batch_12x2d_4x3d", "kind": "batch", "n2": 12, "n3": 4, "lo2": 64, "hi2": 512, "lo3": 32, "hi3": 96, "steps": 4, "mix": 7},
    ]


def _side(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n))


def _sides(rng, lo, hi, most):
    while True:
        s = [_side(rng, lo, hi) for _ in range(3)]
        if s[0] * s[1] * s[2] <= most:
            return {"nx": s[0], "ny": s[1], "nz": s[2]}


def draw(rng):
    kind = rng.choice(["advect", "advect", "solve", "solve", "solve", "step", "step", "flip_splat", "flip_cycle",
                       "extrapolate", "batch"])
    if kind == "advect":
        grid = rng.choice(["density", "velocity", "levelset"])
        return {"kind": kind, "grid": grid, "order": 1 if grid == "levelset" else 2, **_sides(rng, 48, 256, 256 ** 3)}
    if kind == "solve":
        scene, pc, lo, hi = rng.choice([("smoke", "mic", 32, 96), ("liquid", "mic", 48, 128),
                                        ("obstacle", "mgstatic", 64, 224), ("smoke", "mgstatic", 64, 224)])
        return {"kind": kind, "scene": scene, "pc": pc, **_sides(rng, lo, hi, 192 ** 3)}
    if kind == "step":
        if rng.random() < 0.5:
            return {"kind": kind, "pc": "mic", "nx": _side(rng, 64, 256), "ny": _side(rng, 64, 256), "nz": 1}
        return {"kind": kind, "pc": "mgstatic", **_sides(rng, 64, 224, 192 ** 3)}
    if kind in ("flip_splat", "flip_cycle"):
        return {"kind": kind, "fill": rng.choice(["tank", "dam"]), "ppc": rng.choice([4, 8]),
                "shuffled": rng.random() < 0.5, **_sides(rng, 32, 128, 112 ** 3)}
    if kind == "extrapolate":
        return {"kind": kind, "distance": rng.choice([2, 4, 5]), **_sides(rng, 48, 192, 160 ** 3)}
    return {"kind": kind, "n2": rng.randint(2, 12), "n3": rng.randint(1, 4), "lo2": 64, "hi2": rng.randint(128, 512),
            "lo3": 32, "hi3": rng.randint(40, 96), "steps": rng.randint(2, 4), "mix": rng.randint(0, 999)}


# ------------------------------------------------------ inputs, from the seed
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 2654435761 % (2 ** 63))


def _shape(case):
    return case["nz"], case["ny"], case["nx"]


def _axes(case, dtype=torch.float32):
    nz, ny, nx = _shape(case)
    x = torch.arange(nx, device=DEVICE, dtype=dtype).view(1, 1, nx)
    y = torch.arange(ny, device=DEVICE, dtype=dtype).view(1, ny, 1)
    z = torch.arange(nz, device=DEVICE, dtype=dtype).view(nz, 1, 1)
    return x, y, z


def _obstacles(case, scene):
    """the walls of the domain (and a ball inside), as a mask"""
    nz, ny, nx = _shape(case)
    x, y, z = _axes(case)
    wall = (x == 0) | (x == nx - 1) | (y == 0) | (y == ny - 1)
    if nz > 1:
        wall = wall | (z == 0) | (z == nz - 1)
    if scene == "obstacle":
        r = ((x - 0.52 * nx) / (0.15 * nx)) ** 2 + ((y - 0.45 * ny) / (0.15 * ny)) ** 2 + ((z - 0.5 * nz) / (0.15 * nz)) ** 2
        wall = wall | (r < 1)
    return wall.expand(nz, ny, nx).contiguous()


def _phi(case, g):
    """a dam-break surface: a block of liquid with a wavy top and front"""
    nz, ny, nx = _shape(case)
    x, y, z = _axes(case)
    p = torch.rand(6, generator=g, device=DEVICE) * 6.28
    top = 0.58 * ny + 0.04 * ny * torch.sin(x * (9.0 / nx) + p[0]) * torch.cos(z * (7.0 / nz) + p[1])
    front = 0.45 * nx + 0.05 * nx * torch.sin(y * (8.0 / ny) + p[2]) * torch.cos(z * (5.0 / nz) + p[3])
    return torch.maximum(y + 0.5 - top, x + 0.5 - front).clamp(-4.0, 4.0).expand(nz, ny, nx).contiguous()


def _flags(case, scene, phi=None):
    """closed walls, or an open top over smoke; liquid and air from phi"""
    obs = _obstacles(case, scene)
    nz, ny, nx = _shape(case)
    f = torch.full(_shape(case), FLUID, dtype=torch.int32, device=DEVICE)
    if phi is not None:
        f = torch.where(phi <= 0, FLUID, EMPTY).to(torch.int32)
    f[obs] = OBSTACLE
    if scene in ("smoke", "obstacle"):
        z = slice(1, nz - 1) if nz > 1 else slice(0, 1)
        f[z, ny - 1, 1:nx - 1] = OUTFLOW | EMPTY
    return f


def _velocity(case, g, flags):
    """a smooth flow without divergence of a cell or two per step, a little of
    it left over from the forces, nothing through the walls; planes u, v, w"""
    nz, ny, nx = _shape(case)
    vel = torch.zeros((3,) + _shape(case), device=DEVICE)
    r = torch.rand((6, 8), generator=g, device=DEVICE)
    x, y, z = _axes(case)
    for q in range(6):
        k = (r[q, :3] * 2 - 1) * (2 + 3 * q) * 3.1416 / max(nx, ny, nz)
        a = r[q, 3:6] * 2 - 1
        if nz == 1:
            k[2], a[0], a[1] = 0, 0, 0
        d = torch.linalg.cross(k, a)
        d = d * (1.4 / (1 + q) / d.norm().clamp_min(1e-6))
        for c in range(3 if nz > 1 else 2):
            off = [0.5, 0.5, 0.5]
            off[c] = 0.0
            vel[c] += d[c] * torch.cos(k[0] * (x + off[0]) + k[1] * (y + off[1]) + k[2] * (z + off[2]) + 6.28 * r[q, 6])
    vel[1] += 0.05 * torch.rand(_shape(case), generator=g, device=DEVICE)
    obs = (flags & OBSTACLE) != 0
    for c, dim in ((0, 2), (1, 1), (2, 0)):
        shut = obs.clone()
        if obs.shape[dim] > 1:
            shut.narrow(dim, 1, obs.shape[dim] - 1).logical_or_(obs.narrow(dim, 0, obs.shape[dim] - 1))
        vel[c][shut] = 0
    return vel


def _density(case, g):
    nz, ny, nx = _shape(case)
    x, y, z = _axes(case)
    r2 = ((x - 0.5 * nx) / (0.16 * nx)) ** 2 + (((z - 0.5 * nz) / (0.16 * nz)) ** 2 if nz > 1 else 0)
    column = torch.exp(-r2) * (1.0 - y / ny)
    return (column * (0.6 + 0.4 * torch.rand(_shape(case), generator=g, device=DEVICE))).contiguous()


def _source(case, g):
    """inflow noise inside the source at the bottom"""
    nz, ny, nx = _shape(case)
    x, y, z = _axes(case)
    inside = ((x - 0.5 * nx) ** 2 + ((z - 0.5 * nz) ** 2 if nz > 1 else 0) < (0.14 * nx) ** 2) & ((y - 0.1 * ny).abs() < 0.03 * ny + 1)
    return torch.rand(_shape(case), generator=g, device=DEVICE) * inside


def _scene_of(case):
    return {"advect": "closed", "extrapolate": "liquid", "step": "smoke"}.get(case["kind"], case.get("scene"))


def _fields(case, seed):
    """everything a grid case takes, as tensors on the GPU"""
    g = _gen(seed)
    scene = _scene_of(case)
    phi = _phi(case, g) if scene == "liquid" or case.get("grid") == "levelset" else None
    flags = _flags(case, scene, phi)
    out = {"flags": flags, "phi": phi, "vel": _velocity(case, g, flags)}
    if case["kind"] == "step" or case.get("grid") == "density":
        out["density"] = _density(case, g)
    if case["kind"] == "step":
        out["source"] = _source(case, g)
    return out


def _particles(case, seed):
    """particles jittered inside their cells, cell by cell or mixed; flags and
    the two velocity grids beside them"""
    g = _gen(seed)
    nz, ny, nx = _shape(case)
    hx, hy = (nx - 1, ny - 1) if case["fill"] == "tank" else (max(2, int(0.45 * nx)), max(2, int(0.6 * ny)))
    i = torch.arange(1, hx, device=DEVICE)
    j = torch.arange(1, hy, device=DEVICE)
    k = torch.arange(1, nz - 1, device=DEVICE)
    kk, jj, ii = torch.meshgrid(k, j, i, indexing="ij")
    cells = torch.stack([ii, jj, kk], -1).reshape(-1, 3).float()
    pos = cells.repeat_interleave(case["ppc"], 0)
    pos += torch.rand(pos.shape, generator=g, device=DEVICE) * 0.999
    pv = torch.randn(pos.shape, generator=g, device=DEVICE) * 0.3
    pv[:, 0] += torch.sin(pos[:, 1] * (6.0 / ny))
    if case["shuffled"]:
        order = torch.randperm(len(pos), generator=g, device=DEVICE)
        pos, pv = pos[order], pv[order]
    flags = torch.full(_shape(case), EMPTY, dtype=torch.int32, device=DEVICE)
    flags[1:nz - 1, 1:hy, 1:hx] = FLUID
    flags[_obstacles(case, "liquid")] = OBSTACLE
    out = {"flags": flags, "pos": pos.contiguous(), "pv": pv.contiguous()}
    if case["kind"] == "flip_cycle":
        out["vel"] = _velocity(case, g, flags)
        out["velOld"] = out["vel"] * 0.97
    return out


def _batch_scenes(case):
    r = np.random.default_rng(case["mix"])
    sizes = [(int(round(np.exp(r.uniform(np.log(case["lo2"]), np.log(case["hi2"]))))),) * 2 + (1,) for _ in range(case["n2"])]
    sizes += [(int(r.integers(case["lo3"], case["hi3"] + 1)),) * 3 for _ in range(case["n3"])]
    grav = [(0.0, -float(v), 0.0) for v in r.uniform(1e-3, 8e-3, len(sizes))]
    return sizes, grav


# --------------------------------------------------------- prepare, run, work
def _put(grid, t):
    a = t.movedim(0, -1).contiguous() if t.dim() == 4 else t
    m.copyArrayToGridReal(a.cpu().numpy(), grid)
    return grid


class _Buffer:
    """device storage of a grid, for torch"""

    def __init__(self, pointer, shape, kind):
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape, "typestr": kind, "version": 3,
                                         "strides": None, "stream": None}


def _out(state, grid):
    """the grid's storage as a tensor (three planes for vectors)"""
    data, stream = ctypes.c_void_p(), ctypes.c_void_p()
    _lib.check(_lib.load().mg_grid_device(grid._h, ctypes.byref(data), ctypes.byref(stream)))
    vector = isinstance(grid, (m.MACGrid, m.VecGrid))
    key = (data.value, vector)
    if key not in state["views"]:
        nx, ny, nz = state["s"]._size
        shape = (3, nz, ny, nx) if vector else (nz, ny, nx)
        state["views"][key] = torch.as_tensor(_Buffer(data.value, shape, "<f4"), device="cuda")
    view = state["views"][key].detach()
    view.owner = state  # the solver owns the memory: it lives as long as a result does
    return view


PC = {"mic": m.PcMIC, "mgstatic": m.PcMGStatic}


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "views": {}}
    if kind == "batch":
        sizes, grav = _batch_scenes(case)
        state["batch"] = b = mb.BatchedPlumes(sizes, grav, [int(seed) * 1000 + 17 * q + 1 for q in range(len(sizes))])
        for _ in range(2):  # out of rest
            b.step()
        return state
    s = state["s"] = m.Solver(name="perf", gridSize=m.vec3(case["nx"], case["ny"], case["nz"]), dim=3 if case["nz"] > 1 else 2)
    s.timestep = 1.0
    state["flags"] = flags = s.create(m.FlagGrid)
    if kind in ("flip_splat", "flip_cycle"):
        t = _particles(case, seed)
        _put(flags, t["flags"])
        state["parts"] = parts = s.create(m.BasicParticleSystem)
        parts.setPositions(t["pos"].cpu().numpy())
        state["pv"] = parts.create(m.PdataVec3)
        m.copyArrayToPdataVec3(t["pv"].cpu().numpy(), state["pv"])
        for name in ("newVel", "newOld", "weight"):
            state[name] = s.create(m.MACGrid)
        if kind == "flip_cycle":
            state["vel"] = _put(s.create(m.MACGrid), t["vel"])
            state["velOld"] = _put(s.create(m.MACGrid), t["velOld"])
        s.sync()
        return state
    t = _fields(case, seed)
    _put(flags, t["flags"])
    state["vel"] = vel = _put(s.create(m.MACGrid), t["vel"])
    if t["phi"] is not None:
        state["phi"] = _put(s.create(m.LevelsetGrid), t["phi"])
    if "density" in t:
        state["density"] = _put(s.create(m.RealGrid), t["density"])
    if kind == "step":
        # the saved frame that every pass steps on from
        state["density0"] = _put(s.create(m.RealGrid), t["density"])
        state["vel0"] = _put(s.create(m.MACGrid), t["vel"])
        state["source"] = _put(s.create(m.RealGrid), t["source"])
    if kind in ("solve", "step"):
        state["pressure"] = s.create(m.RealGrid)
    if kind == "solve":
        state["rhs"] = s.create(m.RealGrid)
        m.computePressureRhs(rhs=state["rhs"], vel=vel, pressure=state["pressure"], flags=flags, phi=state.get("phi"))
    s.sync()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    flags = state.get("flags")
    if kind == "advect":
        vel = state["vel"]
        grid = vel if case["grid"] == "velocity" else state["density" if case["grid"] == "density" else "phi"]
        m.advectSemiLagrange(flags=flags, vel=vel, grid=grid, order=case["order"])
        return _out(state, grid)
    if kind == "solve":
        m.solvePressureSystem(rhs=state["rhs"], vel=state["vel"], pressure=state["pressure"], flags=flags,
                              phi=state.get("phi"), preconditioner=PC[case["pc"]])
        return _out(state, state["pressure"])
    if kind == "step":
        density, vel, pressure = state["density"], state["vel"], state["pressure"]
        density.copyFrom(state["density0"])
        vel.copyFrom(state["vel0"])
        density.join(state["source"])
        m.advectSemiLagrange(flags=flags, vel=vel, grid=density, order=2, clampMode=2)
        m.advectSemiLagrange(flags=flags, vel=vel, grid=vel, order=2, clampMode=2)
        m.setWallBcs(flags=flags, vel=vel)
        m.addBuoyancy(density=density, vel=vel, gravity=m.vec3(0, -4e-3, 0), flags=flags)
        m.solvePressure(flags=flags, vel=vel, pressure=pressure, cgAccuracy=1e-3, preconditioner=PC[case["pc"]])
        return [_out(state, density), _out(state, vel), _out(state, pressure)]
    if kind in ("flip_splat", "flip_cycle"):
        if kind == "flip_cycle":
            m.flipVelocityUpdate(flags=flags, vel=state["vel"], velOld=state["velOld"], parts=state["parts"],
                                 partVel=state["pv"], flipRatio=0.95)
        m.mapPartsToMAC(flags=flags, vel=state["newVel"], velOld=state["newOld"], parts=state["parts"],
                        partVel=state["pv"], weight=state["weight"])
        return [_out(state, state["newVel"]), _out(state, state["weight"])]
    if kind == "extrapolate":
        m.extrapolateMACSimple(flags=flags, vel=state["vel"], distance=case["distance"])
        m.extrapolateLsSimple(phi=state["phi"], distance=case["distance"])
        return [_out(state, state["vel"]), _out(state, state["phi"])]
    b = state["batch"]
    for _ in range(case["steps"]):
        b.step()
    return [[b.download(q, mb.DENSITY), b.download(q, mb.VELOCITY)] for q in range(len(b))]


def _count_particles(case):
    nz, ny, nx = _shape(case)
    hx, hy = (nx - 1, ny - 1) if case["fill"] == "tank" else (max(2, int(0.45 * nx)), max(2, int(0.6 * ny)))
    return (hx - 1) * (hy - 1) * (nz - 2) * case["ppc"]


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes, _ = _batch_scenes(case)
        n = sum(x * y * z for x, y, z in sizes)
        # per step: density and velocity in and out, flags, source
        return {"bytes": case["steps"] * n * (16 + 16 + 4 + 4), "flops": case["steps"] * n * 300}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "advect":
        if case["grid"] == "velocity":
            return {"bytes": n * (12 + 4 + 12), "flops": n * 3 * 2 * 45}
        return {"bytes": n * (12 + 4 + 4 + (4 if case["order"] == 2 else 0)), "flops": n * case["order"] * 45}
    if kind == "solve":
        return {"bytes": n * (4 + 4 + 4 + (4 if case["scene"] == "liquid" else 0)), "flops": n * 30}
    if kind == "step":  # frame and source in, flags; frame and pressure out
        return {"bytes": n * (16 + 4 + 4 + 16 + 4), "flops": n * 400}
    if kind == "extrapolate":
        return {"bytes": n * (12 + 12 + 4 + 4 + 4), "flops": n * 12}
    p = _count_particles(case)
    cycle = kind == "flip_cycle"  # positions, flags, values; grids in; values and grids out
    return {"bytes": p * (16 + 12 + (12 if cycle else 0)) + n * (36 + (24 if cycle else 0)), "flops": p * 3 * (40 + (60 if cycle else 0))}


# -------------------------------------------------- the same in 64 bits, torch
def _weights(p, n):
    i = p.long()
    s1 = p - i
    s1 = torch.where(p < 0, 0.0, s1)
    i = torch.where(p < 0, 0, i)
    s1 = torch.where(i >= n - 1, 1.0, s1)
    return torch.where(i >= n - 1, n - 2, i), 1 - s1, s1


def _corners(shape, x, y, z):
    """(index, weight) of the up to eight corners of grid positions x, y, z"""
    nz, ny, nx = shape
    xi, s0, s1 = _weights(x, nx)
    yi, t0, t1 = _weights(y, ny)
    base = xi + nx * yi
    layers = [(base, 1.0)]
    if nz > 1:
        zi, f0, f1 = _weights(z, nz)
        base = base + nx * ny * zi
        layers = [(base, f0), (base + nx * ny, f1)]
    for b, f in layers:
        yield b, s0 * t0 * f
        yield b + 1, s1 * t0 * f
        yield b + nx, s0 * t1 * f
        yield b + nx + 1, s1 * t1 * f


def _sample(a, x, y, z):
    flat = a.reshape(-1)
    return sum(flat[i] * w for i, w in _corners(a.shape, x, y, z))


def _inner(a, dx=0, dy=0, dz=0):
    nz, ny, nx = a.shape
    z = slice(1 + dz, nz - 1 + dz) if nz > 1 else slice(0, 1)
    return a[z, 1 + dy:ny - 1 + dy, 1 + dx:nx - 1 + dx]


def _inner_axes(case):
    x, y, z = _axes(case, torch.float64)
    nz, ny, nx = _shape(case)
    return x[..., 1:nx - 1], y[:, 1:ny - 1], z[1:nz - 1] if nz > 1 else z


def _trace_velocity(case, vel, at):
    """velocity at cell centres (at None) or at the faces of component `at`"""
    nz = case["nz"]
    unit = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    out = []
    for c in range(3):
        if c == 2 and nz == 1:
            out.append(torch.zeros_like(_inner(vel[0])))
        elif at is None:
            out.append(0.5 * (_inner(vel[c]) + _inner(vel[c], *unit[c])))
        elif c == at:
            out.append(_inner(vel[c]))
        else:
            d, e = unit[c], tuple(-v for v in unit[at])
            both = tuple(p + q for p, q in zip(d, e))
            out.append(0.25 * (_inner(vel[c]) + _inner(vel[c], *e) + _inner(vel[c], *d) + _inner(vel[c], *both)))
    return out


def _traced(case, v, src, sign):
    x, y, z = _inner_axes(case)
    out = torch.zeros_like(src)
    _inner(out).copy_(_sample(src, x - sign * v[0], y - sign * v[1], z - sign * v[2]))
    return out


def _advected(case, flags, vel, src, order, at):
    """semi-Lagrangian (order 1) or MacCormack with the revert clamp; `at`: a
    velocity component, or None for a cell-centred grid"""
    v = _trace_velocity(case, vel, at)
    fwd = _traced(case, v, src, 1.0)
    if order == 1:
        return fwd
    bwd = _traced(case, v, fwd, -1.0)
    fluid = (flags & FLUID) != 0
    open_ = (flags & (FLUID | EMPTY)) != 0
    fix = fluid.clone()
    if at is not None:
        dim = 2 - at
        n = fluid.shape[dim]
        fix.narrow(dim, 1, n - 1).logical_and_(fluid.narrow(dim, 0, n - 1))
    new = torch.where(fix, fwd + 0.5 * (src - bwd), fwd)
    nz, ny, nx = src.shape
    x, y, z = _inner_axes(case)
    i0 = (x - v[0]).long().clamp(0, nx - 2)
    j0 = (y - v[1]).long().clamp(0, ny - 2)
    k0 = (z - v[2]).long().clamp(0, max(0, nz - 2))
    base = i0 + nx * (j0 + ny * k0)
    lo = torch.full_like(base, 3.0e38, dtype=src.dtype)
    hi = -lo
    some = torch.zeros_like(base, dtype=torch.bool)
    flat, fl = src.reshape(-1), open_.reshape(-1)
    for off in [a + b + c for c in ((0, nx * ny) if nz > 1 else (0,)) for b in (0, nx) for a in (0, 1)]:
        s = flat[base + off]
        ok = fl[base + off] if at is None else torch.ones_like(some)
        lo = torch.where(ok, torch.minimum(lo, s), lo)
        hi = torch.where(ok, torch.maximum(hi, s), hi)
        some |= ok
    keep = some & (_inner(new) >= lo) & (_inner(new) <= hi)
    if at is not None:
        unit = [0, 0, 0]
        unit[at] = -1
        keep &= _inner(open_) & _inner(open_, *unit)
    _inner(new).copy_(torch.where(keep, _inner(new), _inner(fwd)))
    return new


def _solved(case, flags, vel, phi):
    """the solution of the pressure system itself, by conjugate gradients"""
    fluid = (flags & FLUID) != 0
    obs = (flags & OBSTACLE) != 0
    empty = (flags & EMPTY) != 0
    dims = (2, 1, 0) if case["nz"] > 1 else (2, 1)
    inside = torch.zeros_like(fluid)
    _inner(inside).fill_(True)
    live = fluid & inside

    def shifted(a, dim, by):
        return torch.roll(a, -by, dim)

    diag = torch.zeros(flags.shape, dtype=torch.float64, device=flags.device)
    rhs = torch.zeros_like(diag)
    for c, dim in enumerate(dims):
        rhs += vel[c] - shifted(vel[c], dim, 1)
        for by in (1, -1):
            diag += (~shifted(obs, dim, by)).double()
            if phi is not None:
                den = phi - shifted(phi, dim, by)
                theta = torch.where(den > -1e-4, 0.5, (phi / den).clamp(0, 1))
                gf = torch.where(theta < 1e-4, 1e-4, 1 - 1 / theta.clamp_min(1e-30))
                diag -= torch.where(shifted(empty, dim, by), gf, 0.0)
    diag, rhs = torch.where(live, diag, 0.0), torch.where(live, rhs, 0.0)
    links = [(dim, by, (live & shifted(fluid, dim, by)).double()) for dim in dims for by in (1, -1)]

    def apply(a):
        out = diag * a
        for dim, by, w in links:
            out -= w * shifted(a, dim, by)
        return out

    inv = torch.where(live & (diag != 0), 1 / diag, 0.0)
    p, r = torch.zeros_like(rhs), rhs.clone()
    zr = inv * r
    s, sigma = zr.clone(), (zr * r).sum()
    for it in range(4000):
        t = apply(s)
        alpha = sigma / (t * s).sum()
        p += alpha * s
        r -= alpha * t
        if it % 25 == 24 and float(r.abs().max()) < 1e-9:
            break
        zr = inv * r
        new = (zr * r).sum()
        s = zr + (new / sigma) * s
        sigma = new
    return p


def _extrapolated_mac(case, flags, vel, distance):
    fluid, obs = (flags & FLUID) != 0, (flags & OBSTACLE) != 0
    vel = vel.clone()
    nz, ny, nx = flags.shape
    unit = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    near = [s for u in unit for s in (u, tuple(-v for v in u))]
    for c in range(3):
        mark = torch.zeros_like(flags)
        _inner(mark).copy_(_inner(fluid) | _inner(fluid, *(-v for v in unit[c])))
        for d in range(1, distance + 1):
            total = torch.zeros_like(_inner(vel[c]))
            count = torch.zeros_like(total)
            for s in near:
                ok = _inner(mark, *s) == d
                total += torch.where(ok, _inner(vel[c], *s), 0.0)
                count += ok
            hit = (_inner(mark) == 0) & (count > 0)
            _inner(vel[c]).copy_(torch.where(hit, total / count.clamp_min(1), _inner(vel[c])))
            _inner(mark).masked_fill_(hit, d + 1)
    old, new = vel.clone(), torch.zeros_like(vel)
    count = torch.zeros_like(vel[0])
    for c, dim in ((0, 2), (1, 1), (2, 0)):
        n = flags.shape[dim]
        for at, inner, sign in ((0, 1, 1.0), (n - 1, n - 2, -1.0)):
            for q in range(3):
                side = old[q].select(dim, inner).clone()
                if q == c:
                    side = torch.where(obs.select(dim, at) & (sign * side < 0), 0.0, side)
                new[q].select(dim, at).copy_(side)
            count.select(dim, at).add_(1)
    return torch.where(count > 0, new / count.clamp_min(1), vel)


def _extrapolated_phi(case, phi, distance):
    phi = phi.clone()
    mark = torch.zeros(phi.shape, dtype=torch.int32, device=phi.device)
    near = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
    _inner(mark).copy_(_inner(phi) < 0)
    for d in range(1, distance + 1):
        total = torch.zeros_like(_inner(phi))
        count = torch.zeros_like(total)
        for s in near:
            ok = _inner(mark, *s) == d
            total += torch.where(ok, _inner(phi, *s), 0.0)
            count += ok
        hit = (_inner(mark) == 0) & (count > 0)
        if d > 1:
            _inner(phi).copy_(torch.where(hit, total / count.clamp_min(1) + 1.0, _inner(phi)))
        _inner(mark).masked_fill_(hit, d + 1)
    _inner(phi).masked_fill_(_inner(mark) == 0, float(distance + 2))
    return phi


def _splatted(case, pos, pv):
    shape = _shape(case)
    n = shape[0] * shape[1] * shape[2]
    vel, weight = [], []
    for c in range(3):
        v = torch.zeros(n, dtype=torch.float64, device=pos.device)
        w = torch.zeros_like(v)
        off = [0.5, 0.5, 0.5]
        off[c] = 0.0
        for i, q in _corners(shape, *(pos[:, a] - off[a] for a in range(3))):
            w.index_add_(0, i, q)
            v.index_add_(0, i, q * pv[:, c])
        w = torch.where(w < 1e-6, 0.0, w)
        vel.append(torch.where(w != 0, v / w, v).view(shape))
        weight.append(w.view(shape))
    return torch.stack(vel), torch.stack(weight)


def _sample_mac(vel, pos):
    out = []
    for c in range(3):
        off = [0.5, 0.5, 0.5]
        off[c] = 0.0
        out.append(_sample(vel[c], *(pos[:, a] - off[a] for a in range(3))))
    return torch.stack(out, -1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":  # solves that stop at a tolerance, step after step
        return None
    if kind in ("flip_splat", "flip_cycle"):
        t = _particles(case, seed)
        pos, pv = t["pos"].double(), t["pv"].double()
        if kind == "flip_cycle":
            v, o = (_sample_mac(t[k].double(), pos) for k in ("vel", "velOld"))
            pv = 0.95 * (pv + v - o) + 0.05 * v
        return list(_splatted(case, pos, pv))
    t = _fields(case, seed)
    flags, vel = t["flags"], t["vel"].double()
    if kind == "advect":
        if case["grid"] == "velocity":
            return torch.stack([_advected(case, flags, vel, vel[c], case["order"], c) for c in range(3)])
        src = t["density"] if case["grid"] == "density" else t["phi"]
        return _advected(case, flags, vel, src.double(), case["order"], None)
    if kind == "solve":
        return _solved(case, flags, vel, None if t["phi"] is None else t["phi"].double())
    if kind == "extrapolate":
        return [_extrapolated_mac(case, flags, vel, case["distance"]),
                _extrapolated_phi(case, t["phi"].double(), case["distance"])]
    # a step: the velocity and pressure come from a solve that stops at a tolerance
    density = torch.maximum(t["density"], t["source"]).double()
    return [_advected(case, flags, vel, density, 2, None), None, None]
