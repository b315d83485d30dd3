"""Timed cases of the liquid step: whole frames of simulation and the stages a
program can call by themselves, through the Python surface and the C-ABI.

A case is a dict of plain values; its ``kind`` says what one pass does:

  scene        the reference's shipped configuration (Config/PureLiquid3D.json)
               through ``Scene``: particles in, steps, particles out
  frame        a seeded dam break: particle state in from pinned memory,
               ``steps`` x (PreStep, Step), the whole particle state out
  batch        several scenes of uneven sizes in asynchronous mode
  to_grid      PreStep + Particle2Grid on resident particles, fields out
  solve        one pressure solve of given grid fields, pressure out
  net_forward  one application of the learned preconditioner's network
  net_backward the gradient of its parameters

``exact`` gives the outputs of the single stages in 64 bits.  Frames have
none: a particle whose cell, sign of the liquid SDF or wall test falls on the
other side of a rounding takes another branch, and the steps amplify it.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

from liquidhairinteration_b200 import abi, scenes
from liquidhairinteration_b200._lib import call
from liquidhairinteration_b200.model import LiquidModel, Scene
from liquidhairinteration_b200.net import LAYERS, LearnedNet, num_params, param_slices

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WEIGHTS = os.path.join(ROOT, "liquidhairinteration_b200", "weights", "fpcg.lhinet")

DENSITY = 1000.0

# Config/PureLiquid3D.json of the reference, as a program hands it to Scene
PURE_LIQUID = {
    "SolverParameter": {"maxIterations": 100, "tolerance": 0.001, "preconditionerType": "Multigrid", "numLevel": 4,
                        "numPreSmooth": 5, "numPostSmooth": 5, "numFinalSmooth": 20, "smoothingFactor": 0.5},
    "LiquidParameter": {"numParticles": 5000, "viscosity": 0.001, "density": 1000.0, "surfaceTension": 0.0728,
                        "correctCycle": 8},
    "dt": 0.01, "gravity": -9.81, "gridDimension": [64, 64, 64],
    "minCoord": [-1.0, -1.0, -1.0], "maxCoord": [1.0, 1.0, 1.0],
}


def listed():
    return [
        # the reference's own configuration: 64^3 cells, 5000 particles, its solver as written; a few
        # kernels' worth of work per launch, so launches and latency count
        {"name": "scene_pure_liquid", "kind": "scene", "n": 64, "particles": 5000, "steps": 4},
        # one 60 fps frame of the dam breaks of this repository's configurations
        {"name": "frame_dam64", "kind": "frame", "nx": 64, "ny": 64, "nz": 64, "layout": "dam", "precision": "mixed",
         "levels": 4, "sweeps": 5, "w": 1.0, "steps": 8},
        {"name": "frame_dam128", "kind": "frame", "nx": 128, "ny": 128, "nz": 128, "layout": "splash",
         "precision": "mixed", "levels": 5, "sweeps": 2, "w": 1.0, "steps": 8},
        {"name": "frame_dam256", "kind": "frame", "nx": 256, "ny": 256, "nz": 256, "layout": "obstacles",
         "precision": "mixed", "levels": 6, "sweeps": 2, "w": 1.1, "steps": 16},
        # a tank whose cell counts are no multiples of anything, in single precision
        {"name": "frame_ragged_fp32", "kind": "frame", "nx": 93, "ny": 70, "nz": 61, "layout": "splash",
         "precision": "fp32", "levels": 4, "sweeps": 2, "w": 1.0, "steps": 4},
        # the double-precision mode a study checks the others against
        {"name": "frame_fp64", "kind": "frame", "nx": 48, "ny": 48, "nz": 48, "layout": "dam", "precision": "fp64",
         "levels": 4, "sweeps": 2, "w": 1.0, "steps": 4},
        # the batched form: eight scenes of uneven sizes stepped together
        {"name": "batch_8", "kind": "batch", "sizes": "32,48,64,96,32,48,64,40", "precision": "mixed", "steps": 4},
        # the particle-to-grid half alone: a full tank, 8 particles a cell
        {"name": "to_grid_128", "kind": "to_grid", "nx": 128, "ny": 128, "nz": 128, "layout": "tank",
         "precision": "fp32"},
        # the pressure solve alone on grid fields, as a program with its own transfers uses it
        {"name": "solve_192", "kind": "solve", "nx": 192, "ny": 192, "nz": 192, "precision": "mixed",
         "precond": "multigrid", "levels": 5, "sweeps": 2},
        # the same with the learned preconditioner and its shipped weights
        {"name": "solve_learned_128", "kind": "solve", "nx": 128, "ny": 128, "nz": 128, "precision": "mixed",
         "precond": "learned", "levels": 5, "sweeps": 2},
        # the network by itself: applied to one residual, and its gradient as training takes it
        {"name": "net_forward_ragged", "kind": "net_forward", "nx": 120, "ny": 94, "nz": 108},
        {"name": "net_backward_64", "kind": "net_backward", "nx": 64, "ny": 64, "nz": 64},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def around(n, lo):
        return max(lo, int(round(n * rng.uniform(0.6, 1.25))))

    kind = rng.choice(["scene", "frame", "frame", "frame", "batch", "to_grid", "solve", "solve", "net_forward",
                       "net_backward"])
    if kind == "scene":
        return {"kind": "scene", "n": size(40, 96), "particles": size(1000, 40000), "steps": rng.randint(1, 6)}
    if kind == "batch":
        return {"kind": "batch", "sizes": ",".join(str(size(24, 96)) for _ in range(rng.randint(3, 8))),
                "precision": "mixed", "steps": rng.randint(2, 4)}
    if kind == "net_forward" or kind == "net_backward":
        n = size(16, 112) if kind == "net_forward" else size(16, 72)
        return {"kind": kind, "nx": n, "ny": around(n, 8), "nz": around(n, 8)}
    cubic = rng.random() < 0.4
    if kind == "to_grid":
        n = size(20, 160)
        return {"kind": "to_grid", "nx": n, "ny": n if cubic else around(n, 16), "nz": n if cubic else around(n, 16),
                "layout": rng.choice(["tank", "dam", "splash"]), "precision": rng.choice(["fp32", "mixed", "fp64"])}
    if kind == "solve":
        if rng.random() < 0.3:  # the diagonal preconditioner takes any grid
            n = size(24, 96)
            return {"kind": "solve", "nx": n, "ny": around(n, 24), "nz": around(n, 24), "precision": "mixed",
                    "precond": "jacobi", "levels": 1, "sweeps": 1}
        n, m, k = (max(32, size(32, 192) // 16 * 16) for _ in range(3))
        return {"kind": "solve", "nx": n, "ny": n if cubic else m, "nz": n if cubic else k, "precision": "mixed",
                "precond": "multigrid", "levels": 4 if n < 100 else 5, "sweeps": rng.choice([2, 3])}
    n = size(16, 200)
    if cubic:
        n = max(16, n // 16 * 16)
    prec = rng.choice(["mixed", "mixed", "fp32", "fp64"])
    if prec == "fp64":
        n = min(n, 64)
    return {"kind": "frame", "nx": n, "ny": n if cubic else around(n, 16), "nz": n if cubic else around(n, 16),
            "layout": rng.choice(["dam", "splash", "obstacles"]), "precision": prec, "levels": 4 if n < 100 else 5,
            "sweeps": rng.choice([2, 2, 5]), "w": 1.0, "steps": rng.randint(1, 8)}


# ------------------------------------------------------------------ inputs
def _dtype(case):
    return torch.float64 if case.get("precision") == "fp64" else torch.float32


def _extent(case):
    """Domain (1, ny/nx, nz/nx): cubic cells of side 1/nx."""
    return tuple(case[k] / case["nx"] for k in ("nx", "ny", "nz"))


def _dt(case):
    return min(1.0 / 480.0, 1.0 / (3.75 * case["nx"]))


def _wall_box(case):
    ext, h = _extent(case), 1.0 / case["nx"]
    return {"kind": abi.BOUNDARY_RECT, "center": tuple(e / 2 for e in ext),
            "half_extent": tuple(e / 2 - h for e in ext), "use_inside": 1}


def _boundary(case):
    """One-cell walls, with the two solid boxes of the 256^3 dam break in the "obstacles" layout."""
    if case["layout"] != "obstacles":
        return [{"kind": abi.BOUNDARY_NONE, "left": 1}, _wall_box(case)]
    ext = _extent(case)
    boxes = [scenes.box(tuple(a * e for a, e in zip(lo, ext)), tuple(a * e for a, e in zip(hi, ext)))
             for lo, hi in (((0.55, 0.0, 0.2), (0.65, 0.3, 0.4)), ((0.55, 0.0, 0.6), (0.65, 0.3, 0.8)))]
    return [{"kind": abi.BOUNDARY_UNION, "left": 1, "right": 2}, _wall_box(case),
            {"kind": abi.BOUNDARY_UNION, "left": 3, "right": 4}, boxes[0], boxes[1]]


def _swirl(x, phase, k, amp):
    """An Arnold-Beltrami-Childress flow and its gradient (n x 3, n x 9: the
    gradient of component a in columns 3a .. 3a + 2)."""
    a, b, c = amp
    sx, sy, sz = (torch.sin(k * x[:, i] + phase[i]) for i in range(3))
    cx, cy, cz = (torch.cos(k * x[:, i] + phase[i]) for i in range(3))
    u = torch.stack([a * sz + c * cy, b * sx + a * cz, c * sy + b * cx], 1)
    o = torch.zeros_like(sx)
    g = torch.stack([o, -c * k * sy, a * k * cz, b * k * cx, o, -a * k * sz, -b * k * sx, c * k * cy, o], 1)
    return u, g


def _particles(case, seed):
    """(positions, velocities, affine) on the GPU: 8 jittered particles in every cell of the layout's
    liquid inside the walls, moving in a swirl with a little noise, as a step in the middle of a run."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h, ext, dt = 1.0 / nx, _extent(case), _dtype(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    X, Y, Z = ((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * h for n in (nx, ny, nz))
    X, Y, Z = X[:, None, None], Y[None, :, None], Z[None, None, :]
    frac = {"dam": (0.4, 0.6), "splash": (0.4, 0.6), "obstacles": (0.35, 0.7), "tank": (0.95, 0.85)}[case["layout"]]
    wet = ((X < frac[0] * ext[0]) & (Y < frac[1] * ext[1])).expand(nx, ny, nz).clone()
    if case["layout"] == "splash":
        r = 0.15 * min(ext)
        wet |= (X - 0.7 * ext[0]) ** 2 + (Y - 0.7 * ext[1]) ** 2 + (Z - 0.5 * ext[2]) ** 2 < r * r
    inner = torch.zeros_like(wet)
    inner[1:-1, 1:-1, 1:-1] = True
    cell = (wet & inner).nonzero()
    sub = torch.tensor([[a, b, c] for a in (0.25, 0.75) for b in (0.25, 0.75) for c in (0.25, 0.75)], device="cuda",
                       dtype=dt)
    pos = (cell[:, None, :].to(dt) + sub[None]).reshape(-1, 3)
    pos += (torch.rand(pos.shape, generator=g, device="cuda", dtype=dt) - 0.5) * 0.25
    pos *= h
    phase = torch.rand(3, generator=g, device="cuda", dtype=dt) * (2 * math.pi)
    amp = 0.15 + 0.15 * torch.rand(3, generator=g, device="cuda", dtype=dt)
    vel, aff = _swirl(pos, phase, 3 * math.pi, amp)
    vel += 0.02 * torch.randn(vel.shape, generator=g, device="cuda", dtype=dt)
    aff += 0.1 * torch.randn(aff.shape, generator=g, device="cuda", dtype=dt)
    return pos, vel, aff


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _solver(case, **over):
    p = dict(num_level=case["levels"], num_pre_smooth=case["sweeps"], num_post_smooth=case["sweeps"],
             smoothing_factor=case.get("w", 1.0))
    if case["precision"] == "fp32":
        # x is held in single precision: its true residual stalls above the tolerance, so the solve
        # stops on the recursive residual
        p["true_residual_every"] = 0
    p.update(over)
    return scenes.dam(16).solver_params(**p)


def _model(case, solver):
    grid = abi.make_grid_desc((case["nx"], case["ny"], case["nz"]), (0.0, 0.0, 0.0), _extent(case))
    return LiquidModel.from_params(grid, solver, abi.make_liquid_params(density=DENSITY, gravity=-9.81),
                                   case["precision"])


def _shape(case, field):
    shape = [case["nx"], case["ny"], case["nz"]]
    if field in ("vx", "vy", "vz"):
        shape["xyz".index(field[1])] += 1
    return tuple(shape)


def _particle_state(case, seed, solver):
    m = _model(case, solver)
    nodes = _boundary(case)
    call("lhi_liquid_set_boundary", m._h, abi.boundary_array(nodes), len(nodes), 0)
    pos, vel, _ = (_pinned(t) for t in _particles(case, seed))
    n = pos.shape[0]
    out = [torch.empty((n, k), dtype=pos.dtype, pin_memory=True) for k in (3, 3, 9)]
    return {"m": m, "pos": pos, "vel": vel, "out": out, "dt": _dt(case)}


def _subcase(case, n):
    """Scene of the batched form with an n^3 grid."""
    return {"nx": n, "ny": n, "nz": n, "layout": "splash" if n % 3 == 0 else "dam", "precision": case["precision"],
            "levels": 4 if n <= 64 else 5, "sweeps": 2}


def _fields(case, seed):
    """Grid inputs of a pressure solve: the liquid SDF of a wavy pool with a drop above it, open face
    fractions (closed walls and a stepped bed) and face velocities, as float32 on the GPU."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h, ext = 1.0 / nx, _extent(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    ph = torch.rand(6, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)

    def coords(shape, off):
        return [((torch.arange(s, device="cuda", dtype=torch.float64) + o) * h).reshape([-1 if i == a else 1
                                                                                         for i in range(3)])
                for a, (s, o) in enumerate(zip(shape, off))]

    x, y, z = coords((nx, ny, nz), (0.5, 0.5, 0.5))
    level = ext[1] * (0.55 + 0.05 * torch.sin(7 * x + ph[0]) * torch.cos(5 * z + ph[1]))
    r = 0.12 * min(ext)
    drop = torch.sqrt((x - 0.6 * ext[0]) ** 2 + (y - 0.82 * ext[1]) ** 2 + (z - 0.45 * ext[2]) ** 2) - r
    phi = torch.minimum(y - level, drop)
    phi = phi + 0.3 * h * (torch.rand(phi.shape, generator=g, device="cuda", dtype=torch.float64) - 0.5)
    f = {"liquidPhi": None}
    open_cell = torch.zeros((nx, ny, nz), device="cuda", dtype=torch.bool)
    for a, name in enumerate("xyz"):
        shape = [nx, ny, nz]
        shape[a] += 1
        off = [0.5, 0.5, 0.5]
        off[a] = 0.0
        x, y, z = coords(shape, off)
        # a sloped bed cut into steps of 8 cells: its faces are closed, the ones above it open
        bed = 0.2 * ext[1] * (1 - x / ext[0])
        w = (y > (bed / (8 * h)).floor() * (8 * h)).double().expand(shape)
        inner = torch.zeros(shape, device="cuda", dtype=torch.bool)
        lo = [1, 1, 1]
        hi = [s - 1 for s in shape]
        lo[a] += 1  # the faces between the wall cells and the first cells of the interior are closed
        hi[a] -= 1
        inner[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = True
        w = torch.where(inner, w, torch.zeros_like(w)).float().contiguous()
        f["liquidW" + name] = w
        n = open_cell.shape[a]
        open_cell |= (w.narrow(a, 0, n) > 0) | (w.narrow(a, 1, n) > 0)
        p = torch.stack([c.expand(shape).reshape(-1) for c in (x, y, z)], 1)
        amp = torch.full((3,), 0.2, device="cuda", dtype=torch.float64)
        u = _swirl(p, ph[3:], 3 * math.pi, amp)[0][:, a].reshape(shape)
        u = u + 0.05 * torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
        if a == 1:
            u = u - 9.81 * _dt(case)
        f["v" + name] = u.float().contiguous()
    # no liquid in cells without an open face: their pressure has no value
    phi = torch.where(open_cell, phi, torch.full_like(phi, h))
    f["liquidPhi"] = phi.clamp(-2 * h, 3 * h).float().contiguous()
    return f


def _net_inputs(case, seed):
    """(residual, cell types, solid flags, output gradient): a pool whose
    residual mixes smooth and rough parts, walls one cell thick."""
    shape = (case["nx"], case["ny"], case["nz"])
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    ph = torch.rand(4, generator=g, device="cuda") * (2 * math.pi)
    x, y, z = (torch.arange(s, device="cuda", dtype=torch.float32).reshape([-1 if i == a else 1 for i in range(3)])
               for a, s in enumerate(shape))
    wet = (y < 0.6 * shape[1] + 2.0 * torch.sin(0.11 * x + ph[0]) * torch.cos(0.07 * z + ph[1])).expand(shape).clone()
    solid = torch.ones(shape, device="cuda", dtype=torch.bool)
    solid[1:-1, 1:-1, 1:-1] = False
    wet &= ~solid
    r = torch.sin(0.05 * x + ph[2]) * torch.cos(0.08 * y) * torch.sin(0.06 * z + ph[3])
    r = (r + 0.5 * torch.randn(shape, generator=g, device="cuda")) * wet
    dz = torch.randn(shape, generator=g, device="cuda") * wet
    return r.float(), (wet * 2).to(torch.uint8), solid.to(torch.uint8), dz.float()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scene":
        cfg = {**PURE_LIQUID, "gridDimension": [case["n"]] * 3,
               "LiquidParameter": {**PURE_LIQUID["LiquidParameter"], "numParticles": case["particles"]}}
        scene = Scene(cfg)
        m = scene.GetLiquidModel()
        m.Init()
        pos = m.GetParticleSystem().GetPositions()
        rng = np.random.default_rng(seed)
        # the lattice of Init, falling, with a jitter of half a cell
        pos = pos + rng.uniform(-0.25, 0.25, pos.shape).astype(np.float32) * np.float32(m.dx[0])
        vel = rng.normal(0.0, 0.05, pos.shape).astype(np.float32) + np.array([0.0, -0.5, 0.0], np.float32)
        return {"kind": kind, "scene": scene, "m": m, "pos": pos, "vel": vel, "dt": cfg["dt"], "steps": case["steps"]}
    if kind == "frame":
        return {"kind": kind, "steps": case["steps"], **_particle_state(case, seed, _solver(case))}
    if kind == "batch":
        parts = []
        for k, n in enumerate(int(s) for s in case["sizes"].split(",")):
            sub = _subcase(case, n)
            s = _particle_state(sub, seed * 100 + k, _solver(sub, coarse_operator=abi.COARSE_GALERKIN))
            call("lhi_liquid_set_async", s["m"]._h, 1)
            parts.append(s)
        return {"kind": kind, "steps": case["steps"], "parts": parts}
    if kind == "to_grid":
        m = _model(case, _solver({**case, "levels": 4, "sweeps": 2}))
        nodes = _boundary(case)
        call("lhi_liquid_set_boundary", m._h, abi.boundary_array(nodes), len(nodes), 0)
        m.GetParticleSystem().SetParticles(*(t.cpu().numpy() for t in _particles(case, seed)))
        out = {name: torch.empty(_shape(case, name), dtype=_dtype(case), pin_memory=True)
               for name in ("vx", "vy", "vz", "liquidPhi")}
        return {"kind": kind, "m": m, "out": out, "dt": _dt(case)}
    if kind == "solve":
        learned = case["precond"] == "learned"
        kinds = {"learned": abi.PRECOND_LEARNED, "multigrid": abi.PRECOND_MULTIGRID, "jacobi": abi.PRECOND_JACOBI}
        m = _model(case, _solver(case, preconditioner=kinds[case["precond"]],
                                 max_iterations=2000 if case["precond"] == "jacobi" else 200))
        state = {"kind": kind, "m": m, "dt": _dt(case)}
        if learned:
            state["net"] = LearnedNet()
            state["net"].load(WEIGHTS)
            m.GetSolver().SetNetwork(state["net"])
        for name, t in _fields(case, seed).items():
            m.set_field(name, t.cpu().numpy())
        state["out"] = torch.empty(_shape(case, "pressure"), dtype=torch.float32, pin_memory=True)
        return state
    net = LearnedNet()
    net.load(WEIGHTS)
    return {"kind": kind, "net": net, "in": [t.cpu().numpy() for t in _net_inputs(case, seed)]}


# --------------------------------------------------------------------- run
def _download(m, out):
    call("lhi_liquid_get_particles", m._h, *(_ptr(t) for t in out))


def run(state):
    kind, m = state["kind"], state.get("m")
    if kind == "scene":
        ps = m.GetParticleSystem()
        ps.SetParticles(state["pos"], state["vel"])
        for _ in range(state["steps"]):
            m.PreStep(state["dt"])
            m.Step(state["dt"])
            m.PostStep(state["dt"])
        return ps.GetParticles()
    if kind == "frame":
        m.GetParticleSystem().SetParticles(state["pos"].numpy(), state["vel"].numpy())
        for _ in range(state["steps"]):
            m.PreStep(state["dt"])
            m.Step(state["dt"])
        _download(m, state["out"])
        return state["out"]
    if kind == "batch":
        parts = state["parts"]
        for s in parts:
            s["m"].GetParticleSystem().SetParticles(s["pos"].numpy(), s["vel"].numpy())
        for _ in range(state["steps"]):
            for s in parts:
                s["m"].PreStep(s["dt"])
                s["m"].Step(s["dt"])
            for s in parts:
                s["m"].GetSolver().Stats()
        for s in parts:
            _download(s["m"], s["out"])
        return [s["out"] for s in parts]
    if kind == "to_grid":
        m.PreStep(state["dt"])
        m.Particle2Grid()
        for name, t in state["out"].items():
            call("lhi_liquid_get_field", m._h, abi.FIELD_NAMES[name], 0, _ptr(t))
        return state["out"]
    if kind == "solve":
        m.GetSolver().Solve(DENSITY, state["dt"])
        call("lhi_liquid_get_field", m._h, abi.FIELD_NAMES["pressure"], 0, _ptr(state["out"]))
        return state["out"]
    r, types, solid, dz = state["in"]
    if kind == "net_backward":
        return state["net"].backward(r, types, solid, dz)
    return state["net"].forward(r, types, solid)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: what comes in and goes out once, the particle state read and written once a step, each grid
    field of a step written and read once (three velocity components and their weights, liquid SDF,
    pressure, three face fractions).  Flops: 27 window nodes x 3 components with 4 (P2G) and 8 (G2P, with
    the affine part) operations a particle, 50 a cell of a step's grid passes and 13 (one sweep of the
    7-point operator) x 10 a cell of a solve."""
    kind = case["kind"]
    if kind == "batch":
        w = [work({**_subcase(case, int(n)), "kind": "frame", "steps": case["steps"]}) for n in case["sizes"].split(",")]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    if kind == "scene":
        cells, n, s = case["n"] ** 3, case["particles"], 4
        return {"bytes": case["steps"] * (120 * n + 10 * s * cells) + 84 * n,
                "flops": case["steps"] * (972 * n + 180 * cells)}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind in ("net_forward", "net_backward"):
        macs = sum(27 * cin * cout / 8 ** lev for (cin, cout), lev in zip(LAYERS, (0, 1, 2, 1, 0, 0)))
        if kind == "net_forward":
            return {"bytes": 10 * cells + 4 * num_params(), "flops": 2 * macs * 0.6 * cells}
        return {"bytes": 10 * cells + 8 * num_params(), "flops": 6 * macs * 0.6 * cells}
    s = 8 if case["precision"] == "fp64" else 4
    if kind == "solve":
        return {"bytes": 8 * s * cells, "flops": 130 * 0.55 * cells}
    fill = {"dam": 0.24, "splash": 0.25, "obstacles": 0.245, "tank": 0.8}[case["layout"]]
    n = 8 * fill * cells
    if kind == "to_grid":
        return {"bytes": 15 * s * n + 4 * s * cells, "flops": 324 * n + 50 * cells}
    return {"bytes": case["steps"] * (30 * s * n + 10 * s * cells) + 21 * s * n,
            "flops": case["steps"] * (972 * n + 180 * cells)}


# ------------------------------------------------------------------- exact
def _weights64(d):
    """Quadratic B-spline of the distances d (in cells)."""
    d = d.abs()
    return torch.where(d < 0.5, 0.75 - d * d, torch.where(d < 1.5, 0.5 * (1.5 - d) ** 2, torch.zeros_like(d)))


def _exact_to_grid(case, seed):
    pos, vel, aff = (t.double() for t in _particles(case, seed))
    n = (case["nx"], case["ny"], case["nz"])
    h = torch.tensor([e / k for e, k in zip(_extent(case), n)], device="cuda", dtype=torch.float64)
    gpos = pos / h
    cell = gpos.floor().long()
    out = {}
    for a in range(3):
        shape = list(_shape(case, "v" + "xyz"[a]))
        sums = torch.zeros((2, shape[0] * shape[1] * shape[2]), device="cuda", dtype=torch.float64)
        shift = torch.tensor([0.0 if i == a else 0.5 for i in range(3)], device="cuda", dtype=torch.float64)
        for o in ((i, j, k) for i in range(-1, 3) for j in range(-1, 3) for k in range(-1, 3)):
            if any(o[i] == 2 and i != a for i in range(3)):
                continue
            node = cell + torch.tensor(o, device="cuda")
            at = node.double() + shift
            w = _weights64(gpos - at).prod(1)
            val = vel[:, a] + (aff[:, 3 * a:3 * a + 3] * (pos - at * h)).sum(1)
            ok = w > 0
            for i in range(3):
                ok &= (node[:, i] >= 0) & (node[:, i] < shape[i])
            idx = ((node[:, 0] * shape[1] + node[:, 1]) * shape[2] + node[:, 2])[ok]
            sums[0].index_add_(0, idx, w[ok])
            sums[1].index_add_(0, idx, (w * val)[ok])
        v = torch.where(sums[0] < 1e-8, torch.zeros_like(sums[0]), sums[1] / sums[0].clamp_min(1e-300))
        out["v" + "xyz"[a]] = v.reshape(shape)
    # liquid SDF: the nearest particle's distance minus its radius (two cells), over the window of cells
    # within two of the particle's, capped at three cells
    phi = torch.full((n[0] * n[1] * n[2],), float(3 * h[0]), device="cuda", dtype=torch.float64)
    for o in ((i, j, k) for i in range(-2, 3) for j in range(-2, 3) for k in range(-2, 3)):
        c = cell + torch.tensor(o, device="cuda")
        ok = torch.ones(c.shape[0], device="cuda", dtype=torch.bool)
        for i in range(3):
            ok &= (c[:, i] >= 0) & (c[:, i] < n[i])
        d = (pos[ok] - (c[ok].double() + 0.5) * h).norm(dim=1) - 2 * h[0]
        idx = (c[ok, 0] * n[1] + c[ok, 1]) * n[2] + c[ok, 2]
        phi.scatter_reduce_(0, idx, d, "amin")
    out["liquidPhi"] = phi.reshape(n)
    return out


def _exact_solve(case, seed):
    """The ghost-fluid pressure system of the same float32 fields, by conjugate gradients to 1e-13."""
    f = {k: t.double() for k, t in _fields(case, seed).items()}
    h, dt = 1.0 / case["nx"], _dt(case)
    phi = f["liquidPhi"]
    fluid = phi < 0
    diag, b = torch.zeros_like(phi), torch.zeros_like(phi)
    coef = []  # of the face between cell i and i + 1 along each axis, where both cells are fluid
    for a, name in enumerate("xyz"):
        w, v = f["liquidW" + name], f["v" + name]
        m = phi.shape[a]
        b -= (w * v).narrow(a, 1, m) / h - (w * v).narrow(a, 0, m) / h
        t = w.narrow(a, 1, m - 1) * dt / (DENSITY * h * h)
        lo, hi = phi.narrow(a, 0, m - 1), phi.narrow(a, 1, m - 1)
        for c, o, sl in ((lo, hi, 0), (hi, lo, 1)):
            theta = torch.where(o < 0, torch.ones_like(c), (c / (c - o)).clamp_min(0.1))
            diag.narrow(a, sl, m - 1).add_(t / theta)
        coef.append(torch.where((lo < 0) & (hi < 0), t, torch.zeros_like(t)))
    act = fluid & (diag > 0)
    b = torch.where(act, b, torch.zeros_like(b))
    inv = torch.where(act, 1.0 / diag.clamp_min(1e-300), torch.zeros_like(diag))
    diag = torch.where(act, diag, torch.zeros_like(diag))

    def apply(x):
        y = diag * x
        for a, c in enumerate(coef):
            m = x.shape[a]
            y.narrow(a, 0, m - 1).sub_(c * x.narrow(a, 1, m - 1))
            y.narrow(a, 1, m - 1).sub_(c * x.narrow(a, 0, m - 1))
        return y

    x, r = torch.zeros_like(b), b.clone()
    z = inv * r
    p, rz, stop = z.clone(), (r * z).sum(), 1e-13 * float(b.norm())
    for k in range(6000):
        ap = apply(p)
        alpha = rz / (p * ap).sum()
        x += alpha * p
        r -= alpha * ap
        if k % 20 == 19 and float(r.norm()) <= stop:
            break
        z = inv * r
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_net(case, seed, backward):
    r, types, solid, dz = _net_inputs(case, seed)
    params = torch.from_numpy(np.fromfile(WEIGHTS, np.float32, offset=16)).double().cuda()
    ws = []
    for w, _, shape in param_slices():
        p = params[w].reshape(3, 3, 3, shape[1], shape[2]).permute(3, 4, 0, 1, 2).contiguous()
        ws.append(p.requires_grad_(backward))
    wet = types != 0
    pad = torch.nn.functional.pad
    out, air = pad(solid.bool(), (1,) * 6, value=True), pad(~wet & ~solid.bool(), (1,) * 6, value=False)
    near = []
    for m in (air, out):
        s = torch.zeros_like(wet)
        for a in range(3):
            for d in (0, 2):
                i = [slice(1, -1)] * 3
                i[a] = slice(d, d + wet.shape[a])
                s |= m[tuple(i)]
        near.append(s)
    scale = torch.sqrt((r.double()[wet] ** 2).mean())
    rh = torch.where(wet, r.double() / scale, torch.zeros((), device="cuda", dtype=torch.float64))
    a0 = torch.stack([rh, rh * near[0], rh * near[1], torch.zeros_like(rh)])[None]

    def conv(x, w):  # one product per tap: cuDNN has no fast path for 64 bits
        xp = pad(x[0], (1,) * 6)
        n = x.shape[2:]
        y = 0
        for i in range(3):
            for j in range(3):
                for k in range(3):
                    y = y + torch.einsum("oc,cxyz->oxyz", w[:, :, i, j, k],
                                         xp[:, i:i + n[0], j:j + n[1], k:k + n[2]])
        return y[None]

    def up(x, like):
        y = x.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
        return pad(y, (0, like.shape[4] - y.shape[4], 0, like.shape[3] - y.shape[3], 0, like.shape[2] - y.shape[2]))

    pool = torch.nn.functional.avg_pool3d
    with torch.set_grad_enabled(backward):
        h0 = conv(a0, ws[0])
        h1 = conv(pool(h0, 2), ws[1])
        h2 = conv(pool(h1, 2), ws[2])
        u1 = conv(up(h2, h1), ws[3]) + h1
        u0 = conv(up(u1, h0), ws[4]) + h0
        z = torch.where(wet, scale * conv(u0, ws[5])[0, 0], torch.zeros_like(rh))
        if not backward:
            return z
        grads = torch.autograd.grad((z * dz.double()).sum(), ws)
    flat = torch.zeros_like(params)
    for (w, _, _), g in zip(param_slices(), grads):
        flat[w] = g.permute(2, 3, 4, 0, 1).reshape(-1)
    return flat


def exact(case, seed):
    if case["kind"] == "to_grid":
        return _exact_to_grid(case, seed)
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] in ("net_forward", "net_backward"):
        return _exact_net(case, seed, case["kind"] == "net_backward")
    return None
