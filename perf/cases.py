"""The work a user of the solver has it do, as cases that can be timed and checked.

A frame is `update(2 substeps, dt = 1/60 s, 4 iterations)` from a kept state: the program copies that
state into the solver's device fields, steps, and takes positions and velocities in original order,
as a host program with particles of its own identity does (an optimiser, an environment's reset).
Scenes are the repository's builders at their own sizes or smaller and odd ones; a seed gives the
lattice jitter and the initial velocities.  `exact` is the same computation in 64 bits with plain
torch operations, gradients by torch's automatic differentiation.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from __graft_entry__ import load_package

bp = load_package()
abi = bp.abi

DT, SUBSTEPS, ITERATIONS = 1.0 / 60.0, 2, 4
TEXTBOOK = dict(relaxation=600.0, scorr_k=0.001, scorr_n=4, scorr_dq=0.2, xsph_c=0.01)


def listed():
    return [
        # the smallest call: a handful of fluid in an interactive scene, bound by launches
        {"name": "fluid_12", "kind": "frame", "nx": 12, "ny": 12, "nz": 12, "squeeze": 1.0, "cloth": 0, "cubes": 0,
         "mode": "reference", "grid": 64},
        # the 32,768-particle dam break with its textbook parameters
        {"name": "dam_32k", "kind": "frame", "nx": 32, "ny": 32, "nz": 32, "squeeze": 1.0, "cloth": 0, "cubes": 0,
         "mode": "textbook", "grid": 64},
        # a million particles of fluid alone
        {"name": "fluid_1m", "kind": "frame", "nx": 128, "ny": 64, "nz": 128, "squeeze": 1.0, "cloth": 0, "cubes": 0,
         "mode": "reference", "grid": 64},
        # fluid, a cloth under wind and rigid cubes: the headline scene at its start
        {"name": "mixed_1m", "kind": "frame", "nx": 128, "ny": 64, "nz": 128, "squeeze": 1.0, "cloth": 256, "cubes": 64,
         "mode": "reference", "grid": 64},
        # the same late in a run: the fluid 2.5 times as dense and spread over two periods of the table,
        # the cloth and the cubes lying on it
        {"name": "mixed_late", "kind": "frame", "nx": 348, "ny": 14, "nz": 216, "squeeze": 1.357, "cloth": 256,
         "cubes": 64, "mode": "reference", "grid": 64},
        # an odd, middling mixed scene with textbook parameters
        {"name": "mixed_odd", "kind": "frame", "nx": 61, "ny": 33, "nz": 67, "squeeze": 1.1, "cloth": 67, "cubes": 9,
         "mode": "textbook", "grid": 64},
        # a cloth flag alone: many short launches
        {"name": "flag_128", "kind": "flag", "side": 128},
        # the shape-matching stress test: 4096 bodies, 2 million particles, contacts
        {"name": "pile_4096", "kind": "pile", "bodies": 4096},
        # many uneven scenes in one solver
        {"name": "ensemble_40", "kind": "batch", "scenes": 40, "low": 4096, "high": 131072},
        # one step of an optimisation over a rollout: forward, gradients of state, wind and constraints
        {"name": "adjoint_flag", "kind": "adjoint_flag", "side": 128, "frames": 10, "every": 10},
        # the same for a block of fluid
        {"name": "adjoint_block", "kind": "adjoint_block", "nx": 64, "ny": 32, "nz": 32, "frames": 3, "every": 10},
        # the neighbour search alone, on the caller's own buffers
        {"name": "grid_1m", "kind": "grid", "points": 1000003, "grid": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "flag", "pile", "batch", "adjoint_flag", "adjoint_block",
                       "grid"])
    if kind == "frame":
        total = _log(rng, 600, 1000000)
        nx = max(4, int(round(total ** (1 / 3) * math.exp(rng.uniform(-0.4, 0.4)))))
        ny = max(4, int(round(total ** (1 / 3) * math.exp(rng.uniform(-0.7, 0.1)))))
        nz = max(4, min(400, total // (nx * ny)))
        solids = rng.random() < 0.5
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "squeeze": round(rng.uniform(1.0, 1.3), 3),
                "cloth": _log(rng, 8, 200) if solids else 0, "cubes": rng.choice([1, 4, 16, 25]) if solids else 0,
                "mode": rng.choice(["reference", "textbook"]), "grid": rng.choice([32, 64, 64, 128])}
    if kind == "flag":
        return {"kind": kind, "side": _log(rng, 9, 200)}
    if kind == "pile":
        return {"kind": kind, "bodies": _log(rng, 8, 4000)}
    if kind == "batch":
        return {"kind": kind, "scenes": _log(rng, 2, 48), "low": _log(rng, 500, 5000), "high": _log(rng, 6000, 120000)}
    if kind == "adjoint_flag":
        return {"kind": kind, "side": _log(rng, 9, 140), "frames": rng.randint(2, 10), "every": rng.choice([4, 10])}
    if kind == "adjoint_block":
        n = _log(rng, 8, 36)
        return {"kind": kind, "nx": n + rng.randint(0, 9), "ny": n, "nz": n + rng.randint(0, 5), "frames": 2,
                "every": rng.choice([2, 10])}
    return {"kind": kind, "points": _log(rng, 1000, 2000000), "grid": rng.choice([32, 64, 128, 256])}


# ---- scenes ----------------------------------------------------------------------


@functools.lru_cache(maxsize=32)
def _base(key):
    """The scene(s) of a case before its seed, and the solver parameters."""
    case, sc = dict(key), bp.scenes
    kind = case["kind"]
    if kind in ("frame", "adjoint_block"):
        n = (case["nx"], case["ny"], case["nz"])
        if case.get("cloth"):
            s = sc.mixed_phase_1m(fluid=n, cloth=case["cloth"], cubes=case["cubes"])
        else:
            s = sc.pbf_scene(*n, box=tuple(0.1 * k + 0.8 for k in (n[0], 2 * n[1], n[2])))
        s.grid_dim = case.get("grid", 64)
        squeeze = np.float32(case.get("squeeze", 1.0))
        if squeeze != 1.0:  # a denser fluid, and the solids just above it
            fluid = s.phases < 0
            top = s.positions[fluid, 1].max() / squeeze
            s.positions[fluid] = np.float32(0.1) + (s.positions[fluid] - np.float32(0.1)) / squeeze
            if not fluid.all():
                cloth_y = s.positions[~fluid, 1].min()
                s.positions[~fluid, 1] += top + np.float32(0.09) - cloth_y
                cubes = np.arange(len(fluid)) >= np.flatnonzero(fluid).size + case["cloth"] ** 2
                s.positions[cubes, 1] -= np.float32(1.9)
        if kind == "adjoint_block":
            p = bp.make_params(s, stage_mask=abi.BP_STAGE_FLUID | abi.BP_STAGE_PLANES | abi.BP_STAGE_XSPH)
        elif case["mode"] == "reference":
            p = bp.make_params(s, mass_scaling_k=0.0)
        else:
            p = bp.make_params(s, mode=abi.BP_MODE_TEXTBOOK, wind_velocity=(3.0, 0.0, 1.0), wind_lift=0.3,
                               wind_drag=1.0, rotation_iterations=10, mass_scaling_k=0.0, **TEXTBOOK)
        return [s], [p]
    if kind in ("flag", "adjoint_flag"):
        s = sc.flag_scene(n=case["side"])
        p = bp.make_params(s, mode=abi.BP_MODE_TEXTBOOK,
                           stage_mask=abi.BP_STAGE_PLANES | abi.BP_STAGE_WIND | abi.BP_STAGE_DISTANCE
                           | abi.BP_STAGE_IMMOVABLE,
                           wind_velocity=(4.0, 0.0, 0.0), wind_drag=1.0, wind_lift=0.3, mass_scaling_k=0.0)
        return [s], [p]
    if kind == "pile":
        side = max(2, math.ceil(math.sqrt(case["bodies"] / 4)))
        s = sc.rigid_body_pile(bodies=case["bodies"], lattice=(side, 4, side))
        return [s], [bp.make_params(s, stage_mask=abi.BP_STAGE_PLANES | abi.BP_STAGE_PARTICLE_COLLISION
                                    | abi.BP_STAGE_SHAPE_MATCHING)]
    scenes = sc.dam_break_ensemble(num_scenes=case["scenes"], lo=case["low"], hi=case["high"])
    return scenes, [bp.make_params(s) for s in scenes]


def _scenes(case):
    return _base(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


def _state(case, seed):
    """Positions and velocities of all scenes' particles, in original order: [N, 3] float32 each."""
    scenes, _ = _scenes(case)
    rng = np.random.default_rng(seed)
    x = np.concatenate([s.positions for s in scenes])
    phase = np.concatenate([s.phases for s in scenes])
    jitter = np.where(phase < 0, 2e-3, 2e-5).astype(np.float32)[:, None]  # 0.01 spacings for fluid
    x = x + (rng.random(x.shape, np.float32) - np.float32(0.5)) * jitter
    v = (rng.random(x.shape, np.float32) - np.float32(0.5)) * np.float32(0.6)
    return x, v, phase


# ---- prepare and run -------------------------------------------------------------


class _Device:
    """Device memory of a solver, which lives as long as a tensor over it does."""

    def __init__(self, solver, ptr, shape, kind):
        self.solver = solver
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 2}


def _fields(solver, before=None):
    """The solver's state as device tensors, valid until its next update (`before`: kept where they did not move)."""
    out = {}
    for name, field, width, kind in (("x", abi.BP_FIELD_POSITIONS, 4, "<f4"), ("v", abi.BP_FIELD_VELOCITIES, 4, "<f4"),
                                     ("id", abi.BP_FIELD_MAP_TO_ORIGINAL, 1, "<i4"),
                                     ("new", abi.BP_FIELD_MAP_TO_NEW, 1, "<i4"),
                                     ("rot", abi.BP_FIELD_RIGID_ROTATIONS, 4, "<f4")):
        ptr, nbytes = solver.field_ptr(field)
        if not nbytes:
            continue
        if before and before[name].data_ptr() == ptr:
            out[name] = before[name]
        else:
            shape = (nbytes // 16, 4) if width == 4 else (nbytes // 4,)
            out[name] = torch.as_tensor(_Device(solver, ptr, shape, kind), device="cuda")
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid":
        gen = torch.Generator("cuda").manual_seed(seed)
        n, D, dev = case["points"], case["grid"], "cuda"
        side = 0.1 * n ** (1 / 3) * 1.3  # fluid-like density, some of the box empty
        pos = torch.rand((n, 3), generator=gen, device=dev) * side
        size = C.c_size_t()
        lib = abi.load()
        abi.check(lib, lib.bp_grid_workspace_size(n, D, C.byref(size)))
        ints = lambda m: torch.empty(m, dtype=torch.int32, device=dev)  # noqa: E731
        return {"kind": kind, "lib": lib, "n": n, "D": D, "pos": pos, "ids": ints(n), "sorted": ints(n),
                "order": ints(n), "start": ints(D ** 3).fill_(-1), "end": ints(D ** 3).fill_(-1), "counts": ints(n),
                "built": False, "work": torch.empty(size.value, dtype=torch.uint8, device=dev), "size": size.value}
    scenes, params = _scenes(case)
    # the solver's own stream, which orders itself with the default stream
    solver = bp.BatchSolver(scenes, params) if kind == "batch" else bp.ParticleSolver(scenes[0], params[0])
    x, v, _ = _state(case, seed)
    solver.set_state(x, v)
    fields = _fields(solver)
    state = {"kind": kind, "solver": solver, "fields": fields,
             "start": {k: fields[k].clone() for k in ("x", "v", "id", "rot") if k in fields}}
    if kind.startswith("adjoint"):
        state.update(frames=case["frames"], every=case["every"], target=_target(case, seed))
    return state


def _target(case, seed):
    """The flag's target pose; None: the loss is the block's centre of mass."""
    if case["kind"] != "adjoint_flag":
        return None
    x = _scenes(case)[0][0].positions
    return x + np.random.default_rng(seed + 7).normal(0.0, 0.05, x.shape).astype(np.float32)


def run(state):
    if state["kind"] == "grid":
        return _run_grid(state)
    solver = state["solver"]
    for k, kept in state["start"].items():
        state["fields"][k].copy_(kept)
    if state["kind"].startswith("adjoint"):
        return _run_adjoint(state, solver)
    if state["kind"] == "batch":
        solver.step(DT, SUBSTEPS, ITERATIONS)
    else:
        solver.update(SUBSTEPS, DT, ITERATIONS)
    f = state["fields"] = _fields(solver, state["fields"])
    out = {"x": f["x"].index_select(0, f["new"])[:, :3], "v": f["v"].index_select(0, f["new"])[:, :3]}
    if "rot" in f:
        out["rot"] = f["rot"]
    return out


def _run_adjoint(state, solver):
    solver.tape_begin(state["every"])
    for _ in range(state["frames"]):
        solver.update(SUBSTEPS, DT, ITERATIONS)
    x = solver.positions()
    if state["target"] is None:
        g = np.full(x.shape, 1.0 / len(x), np.float32)
    else:
        g = (np.float32(2.0 / len(x)) * (x - state["target"])).astype(np.float32)
    out = solver.backward(g)
    solver.tape_end()
    state["fields"] = _fields(solver, state["fields"])
    out = {k: v for k, v in out.items() if v.size and (state["target"] is not None or k in ("positions", "velocities"))}
    return {"x": x, "grad": out}


def _run_grid(s):
    lib, n, D = s["lib"], s["n"], s["D"]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    at = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    if s["built"]:  # the ranges of the last build, as the reference's loop resets them
        abi.check(lib, lib.bp_grid_reset(st, n, at(s["sorted"]), at(s["start"]), at(s["end"])))
    abi.check(lib, lib.bp_grid_build(st, n, at(s["pos"]), C.c_float(0.2), D, at(s["ids"]), at(s["sorted"]),
                                     at(s["order"]), at(s["start"]), at(s["end"]), at(s["work"]),
                                     C.c_size_t(s["size"])))
    s["built"] = True
    pos = s["pos"].index_select(0, s["order"])
    abi.check(lib, lib.bp_grid_neighbor_counts(st, n, at(pos), C.c_float(0.2), D, C.c_float(0.2), at(s["start"]),
                                               at(s["end"]), at(s["counts"])))
    return {"ids": s["ids"], "sorted": s["sorted"], "order": s["order"], "start": s["start"], "end": s["end"],
            "counts": s["counts"]}


def work(case):
    """State in and out, and the pair arithmetic of each particle's neighbours (33.5 within h = 2 spacings at rest)."""
    kind = case["kind"]
    if kind == "grid":
        n = case["points"]
        return {"bytes": 12 * n + 16 * n + 8 * min(n, case["grid"] ** 3), "flops": 33.5 * 8 * n}
    scenes, _ = _scenes(case)
    n = sum(s.num_particles for s in scenes)
    fluid = sum(int((s.phases < 0).sum()) for s in scenes)
    edges = sum(s.num_distance_constraints for s in scenes)
    pairs = 33.5 * case.get("squeeze", 1.0) ** 3 * fluid
    frame = SUBSTEPS * (ITERATIONS * (pairs * 40 + (n - fluid) * 60 + edges * 40) + pairs * 75)
    bytes_ = 36 * n + 36 * n
    if kind.startswith("adjoint"):
        return {"bytes": bytes_ + 24 * n + 8 * edges, "flops": 3 * case["frames"] * frame}
    return {"bytes": bytes_, "flops": frame}


# ---- the same in 64 bits -----------------------------------------------------------


def exact(case, seed):
    if case["kind"] == "grid":
        return None
    scenes, params = _scenes(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, v, _ = _state(case, seed)
    xs, vs, rots, first = [], [], [], 0
    if case["kind"].startswith("adjoint"):
        return _exact_adjoint(case, seed, scenes[0], params[0], x, v, dev)
    with torch.no_grad():
        for s, p in zip(scenes, params):
            m = s.num_particles
            step = _Exact(s, p, dev)
            a = torch.as_tensor(x[first:first + m], device=dev).double()
            b = torch.as_tensor(v[first:first + m], device=dev).double()
            for _ in range(SUBSTEPS):
                a, b = step.substep(a, b)
            xs.append(a)
            vs.append(b)
            rots.append(step.rot)
            first += m
    out = {"x": torch.cat(xs), "v": torch.cat(vs)}
    if len(scenes) == 1 and len(scenes[0].rigid_ranges):
        out["rot"] = rots[0]
    return out


def _exact_adjoint(case, seed, scene, params, x, v, dev):
    step = _Exact(scene, params, dev)
    leaf = lambda t: t.detach().double().requires_grad_()  # noqa: E731
    x0, v0 = leaf(torch.as_tensor(x, device=dev)), leaf(torch.as_tensor(v, device=dev))
    step.wind, step.rest, step.stiff = leaf(step.wind), leaf(step.rest), leaf(step.stiff)
    a, b = x0, v0
    for _ in range(case["frames"] * SUBSTEPS):
        a, b = step.substep(a, b)
    target = _target(case, seed)
    if target is None:
        a.sum().div(len(x)).backward()
        return {"x": a.detach(), "grad": {"positions": x0.grad, "velocities": v0.grad}}
    ((a - torch.as_tensor(target, device=dev).double()) ** 2).sum().div(len(x)).backward()
    return {"x": a.detach(), "grad": {"positions": x0.grad, "velocities": v0.grad, "wind_velocity": step.wind.grad,
                                      "distance_stiffness": step.stiff.grad, "distance_rest_length": step.rest.grad}}


def _dot(a, b):
    return (a * b).sum(-1)


class _Exact:
    """One scene's substep in 64 bits.  The cell of a position is integer work that the solver defines in
    32 bits, so it is taken from the position rounded to 32 bits; everything else is in doubles.  Particles
    keep their original order; `slot` is the place each one has in the cell-sorted order."""

    def __init__(self, scene, p, dev):
        t = lambda a, kind: torch.as_tensor(np.ascontiguousarray(a), device=dev).to(kind)  # noqa: E731
        self.p, self.dev, self.n = p, dev, scene.num_particles
        self.dt = DT / SUBSTEPS
        self.mass, self.phase = t(scene.masses, torch.double), t(scene.phases, torch.long)
        self.fluid = self.phase < 0
        self.planes = t(scene.planes, torch.double)
        self.pairs = t(scene.distance_pairs, torch.long).reshape(-1, 2)
        self.rest = t(scene.distance_params.reshape(-1, 2)[:, 0], torch.double)
        self.stiff = t(scene.distance_params.reshape(-1, 2)[:, 1], torch.double)
        self.faces = t(scene.faces, torch.long).reshape(-1, 3)
        self.pinned = t(scene.immovables, torch.long)
        self.wind = torch.tensor(list(p.wind_velocity), dtype=torch.double, device=dev)
        self.gravity = torch.tensor(list(p.gravity), dtype=torch.double, device=dev)
        self.textbook = p.mode == abi.BP_MODE_TEXTBOOK
        bodies = len(scene.rigid_ranges)
        self.rot = torch.tensor([0.0, 0.0, 0.0, 1.0], dtype=torch.double, device=dev).repeat(bodies, 1)
        if bodies:
            r = t(scene.rigid_ranges, torch.long)
            self.body = torch.repeat_interleave(torch.arange(bodies, device=dev), r[:, 1] - r[:, 0])
            self.member = torch.arange(len(self.body), device=dev) + (
                r[:, 0] - torch.cumsum(r[:, 1] - r[:, 0], 0) + (r[:, 1] - r[:, 0]))[self.body]
            self.shape = t(scene.rigid_rest, torch.double)[self.member]
            self.members = (r[:, 1] - r[:, 0]).double()[:, None]
        h, pi = float(p.kernel_radius), float(np.float32(3.141592))
        self.h, self.h2 = h, h * h
        self.poly6_c, self.spiky_c = 315 / 64 / pi / h ** 9, -45 / pi / h ** 6
        self.akinci_c, self.akinci_off = 32 / pi / h ** 9, h ** 6 / 64
        if self.textbook:
            self.akinci_off *= self.akinci_c

    def on(self, bit):
        return bool(self.p.stage_mask & bit)

    def cells(self, x):
        f = x.detach().float() + 50000.0
        return torch.trunc(f / torch.full_like(f, self.p.cell_size)).long()

    def address(self, c):
        D = self.p.grid_dim
        c = c & (D - 1)
        return c[..., 0] * D * D + c[..., 1] * D + c[..., 2]

    def near(self, x, radius2):
        """Pairs (i, j) of the 27 cells with |x_i - x_j|^2 <= radius2."""
        with torch.no_grad():
            x = x.detach()
            o = torch.tensor([[a, b, c] for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)], device=self.dev)
            found = []
            chunk = max(1, int(4e7) // max(27, int(27 * self.fullest)))
            for i0 in range(0, self.n, chunk):
                a = self.address(self.cells(x[i0:i0 + chunk])[:, None, :] + o)
                b, m = self.off[a].reshape(-1), (self.off[a + 1] - self.off[a]).reshape(-1)
                run = torch.repeat_interleave(torch.arange(len(m), device=self.dev), m)
                k = torch.arange(len(run), device=self.dev) - (torch.cumsum(m, 0) - m)[run] + b[run]
                i, j = run // 27 + i0, self.order[k]
                keep = ((x[i] - x[j]) ** 2).sum(-1) <= radius2
                found.append((i[keep], j[keep]))
            return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])

    def total(self, i, values):
        return torch.zeros((self.n,) + values.shape[1:], dtype=torch.double, device=self.dev).index_add(0, i, values)

    def poly6(self, d2):
        return self.poly6_c * (self.h2 - d2) ** 3

    def spiky(self, diff, d2):
        r = torch.sqrt(d2)
        return (self.spiky_c * (self.h - r) ** 2 / r)[:, None] * diff

    def substep(self, x, v):
        p, dt = self.p, self.dt
        q = x + v * dt + self.gravity * dt * dt
        key = self.address(self.cells(q))
        # ties keep the order of the substep before
        before = getattr(self, "order", torch.arange(self.n, device=self.dev))
        self.order = before[torch.sort(key[before], stable=True).indices]
        self.slot = torch.empty_like(self.order)
        self.slot[self.order] = torch.arange(self.n, device=self.dev)
        count = torch.bincount(key, minlength=p.grid_dim ** 3)
        self.off = torch.cat([torch.zeros(1, dtype=torch.long, device=self.dev), torch.cumsum(count, 0)])
        self.fullest = float((count.double() ** 2).sum() / self.n)
        w = torch.exp(p.mass_scaling_k * x[:, 1] * math.log(float(np.float32(2.7182818284)))) / self.mass
        xs = x
        if self.on(abi.BP_STAGE_PLANES):
            for plane in torch.cat([self.planes, self.planes]):
                d = _dot(plane[:3] - xs, plane[3:]) + p.particle_radius
                move = torch.where(d > 0, d, torch.zeros_like(d))[:, None] * plane[3:]
                xs, q = xs + move, q + move
        if self.on(abi.BP_STAGE_WIND) and len(self.faces):
            q = self.blow(q, v)
        for _ in range(ITERATIONS):
            if self.on(abi.BP_STAGE_PLANES):
                q = self.walls(xs, q)
            if self.on(abi.BP_STAGE_PARTICLE_COLLISION) and not bool(self.fluid.all()):
                q = self.contacts(xs, q, w)
            if self.on(abi.BP_STAGE_FLUID):
                q = self.incompressible(q)
            if self.on(abi.BP_STAGE_DISTANCE) and len(self.pairs):
                i, j = self.pairs[:, 0], self.pairs[:, 1]
                diff = q[i] - q[j]
                d = torch.sqrt(_dot(diff, diff))
                k = diff * ((d - self.rest) / (w[i] + w[j]) * self.stiff / d)[:, None]
                q = q + self.total(i, -w[i][:, None] * k) + self.total(j, w[j][:, None] * k)
            if self.on(abi.BP_STAGE_SHAPE_MATCHING) and len(self.rot):
                q = self.match(q)
            if self.on(abi.BP_STAGE_IMMOVABLE) and len(self.pinned):
                q = q.index_copy(0, self.pinned, xs[self.pinned])
        return q, self.after(q, (q - xs) / dt)

    def walls(self, xs, q):
        p = self.p
        for plane in self.planes:
            n = plane[3:]
            d = _dot(plane[:3] - q, n) + p.particle_radius
            hit = torch.nonzero(d > 0)[:, 0]
            if not len(hit):
                continue
            diff = q[hit] - xs[hit]
            dn = _dot(diff, n)
            side = diff - dn[:, None] * n
            length = torch.sqrt(_dot(side, side).clamp(min=1e-300))
            to = q[hit] + d[hit][:, None] * n
            dx = to - xs[hit]
            slide = dx - _dot(dx, n)[:, None] * n
            part = torch.where(length < p.friction_static * dn, torch.ones_like(dn),
                               (p.friction_dynamic * -dn / length).clamp(max=1.0))
            q = q.index_copy(0, hit, to - slide * part[:, None])
        return q

    def contacts(self, xs, q, w):
        p, r = self.p, self.p.particle_radius
        i, j = self.near(q, 4 * r * r)
        pi, pj = self.phase[i], self.phase[j]
        diff = q[i] - q[j]
        d2 = _dot(diff, diff)
        keep = (pi != pj) & ((pi > 0) | (pj > 0)) & (d2 < 4 * r * r) & (d2 > 1e-5)
        i, j, diff, d2 = i[keep], j[keep], diff[keep], d2[keep]
        d = torch.sqrt(d2)
        w1 = (w[i] / (w[i] + w[j]))[:, None]
        push = diff * (2 * r / d - 1)[:, None]
        dx = w1 * push
        dx2 = _dot(dx, dx)
        slide = (dx + q[i] - xs[i]) - (q[j] - (1 - w1) * push - xs[j])
        nn = diff / d[:, None]
        slide = slide - _dot(slide, nn)[:, None] * nn
        s2 = _dot(slide, slide)
        part = torch.where(s2 <= p.friction_static ** 2 * dx2, torch.ones_like(s2),
                           (p.friction_dynamic * torch.sqrt(dx2 / s2.clamp(min=1e-300))).clamp(max=1.0))
        counted = (dx2 > r * r * 1e-6).double()
        rub = self.total(i, -(w1 * slide) * (part * counted)[:, None])
        return q + self.total(i, dx) + rub / self.total(i, counted).clamp(min=1.0)[:, None]

    def incompressible(self, q):
        p, rho0 = self.p, self.p.rest_density
        akinci = self.on(abi.BP_STAGE_AKINCI)
        i, j = self.near(q, self.h2)
        diff = q[i] - q[j]
        d2 = _dot(diff, diff)
        apart = d2.detach() > 0
        weigh = self.mass[j] * self.poly6(d2) * torch.where(self.fluid[j], 1.0, float(p.solid_density_scale))
        counted = self.fluid[i] if self.textbook else self.fluid[i] & (self.slot[j] >= self.slot[i])
        self.rho = self.total(i[counted], weigh[counted])
        c = self.rho / rho0 - 1
        if akinci:
            c = c.clamp(min=0.0)
        i, j, diff, d2 = i[apart], j[apart], diff[apart], d2[apart]
        grad = self.spiky(diff, d2)
        if self.textbook:
            g = -(self.mass[j] / rho0)[:, None] * grad
            mean = self.total(i, g)
            lam = -c / (self.total(i, _dot(g, g)) + _dot(mean, mean) + p.relaxation)
        else:
            lam = -c / p.lambda_denominator
        lam = torch.where(self.fluid, lam, torch.zeros_like(lam))
        s = lam[i] + lam[j]
        if self.textbook or not akinci:
            s = s - p.scorr_k * (self.poly6(d2) / self.poly6((p.scorr_dq * self.h) ** 2)) ** p.scorr_n
        move = s[:, None] * grad
        if self.textbook:
            moves = self.fluid[i]
        else:
            moves = torch.where(self.slot[j] > self.slot[i], self.fluid[i], self.fluid[j])
            if p.delta_clamp > 0:
                length = torch.sqrt(_dot(move, move).clamp(min=1e-300))
                move = move * (p.delta_clamp / length).clamp(max=1.0)[:, None]
        return q + self.total(i[moves], (self.mass[j][:, None] * move)[moves]) / rho0

    def blow(self, q, v):
        p, (a, b, c) = self.p, self.faces.T
        u = (v[a] + v[b] + v[c]) / 3 - (self.wind if self.textbook else 0.0)
        n = torch.linalg.cross(q[b] - q[a], q[c] - q[a])
        speed, twice = torch.sqrt(_dot(u, u).clamp(min=1e-300)), torch.sqrt(_dot(n, n).clamp(min=1e-300))
        live = ((speed > 1e-5) & (twice > 1e-5)).double()
        uh, n = u / speed[:, None], n / twice[:, None]
        n = torch.where((_dot(n, u) > 0)[:, None], n, -n)
        much = speed * speed * 0.5 * twice * _dot(n, uh) * live
        lift = torch.linalg.cross(torch.linalg.cross(n, uh), uh)
        move = (p.wind_lift * lift - p.wind_drag * uh) * much[:, None] * self.dt ** 2
        for k in (a, b, c):
            q = q + self.total(k, move / self.mass[k][:, None])
        return q

    def match(self, q):
        m = len(self.rot)

        def sums(t):
            return torch.zeros((m,) + t.shape[1:], dtype=torch.double, device=self.dev).index_add(0, self.body, t)

        centre = sums(q[self.member]) / self.members
        A = sums((q[self.member] - centre[self.body])[:, :, None] * self.shape[:, None, :])
        r, live = self.rot, torch.ones(m, dtype=torch.bool, device=self.dev)
        for _ in range(self.p.rotation_iterations):
            R = self.matrix(r)
            om = torch.linalg.cross(R, A, dim=1).sum(2) * (1 / (R * A).sum((1, 2)).abs() + 1e-9)[:, None]
            w2 = _dot(om, om)
            live = live & (w2 > 1e-9)
            wl = torch.sqrt(w2.clamp(min=1e-300))
            ax, half = om / wl[:, None], wl / 2
            a, aw = ax * torch.sin(half)[:, None], torch.cos(half)
            b, bw = r[:, :3], r[:, 3]
            new = torch.cat([aw[:, None] * b + bw[:, None] * a + torch.linalg.cross(a, b),
                             (aw * bw - _dot(a, b))[:, None]], 1)
            r = torch.where(live[:, None], new / torch.sqrt(_dot(new, new))[:, None], r)
        self.rot = r
        goal = (self.matrix(r)[self.body] @ self.shape[:, :, None])[:, :, 0] + centre[self.body]
        return q.index_copy(0, self.member, goal)

    @staticmethod
    def matrix(r):
        x, y, z, w = r.T
        rows = [1 - 2 * y * y - 2 * z * z, 2 * x * y - 2 * w * z, 2 * x * z + 2 * w * y,
                2 * x * y + 2 * w * z, 1 - 2 * x * x - 2 * z * z, 2 * y * z - 2 * w * x,
                2 * x * z - 2 * w * y, 2 * y * z + 2 * w * x, 1 - 2 * x * x - 2 * y * y]
        return torch.stack(rows, 1).reshape(-1, 3, 3)

    def after(self, q, v):
        p = self.p
        swirl, tension, viscous = (self.on(b) for b in (abi.BP_STAGE_VORTICITY, abi.BP_STAGE_AKINCI, abi.BP_STAGE_XSPH))
        if not (swirl or tension or viscous) or not bool(self.fluid.any()):
            return v
        rho = getattr(self, "rho", None)
        i, j = self.near(q, self.h2)
        keep = self.fluid[i] & (self.phase[i] == self.phase[j]) & (i != j)
        i, j = i[keep], j[keep]
        diff = q[i] - q[j]
        d2 = _dot(diff, diff)
        full = (i, j, d2)
        if swirl or tension:
            a = d2.detach() > 0
            i, j, diff, d2 = i[a], j[a], diff[a], d2[a]
            g, r = self.spiky(diff, d2), torch.sqrt(d2)
        if swirl:
            om = self.total(i, torch.linalg.cross(v[j] - v[i], g))
            eta = self.total(i, torch.sqrt(_dot(om, om))[j][:, None] * g)
            e2 = _dot(eta, eta)
            turn = p.vorticity_eps * torch.linalg.cross(eta / torch.sqrt(e2.clamp(min=1e-300))[:, None], om) * self.dt
        if tension:
            nrm = self.h * self.total(i, g / rho[j][:, None])
            t3 = self.akinci_c * ((self.h - r) * r) ** 3
            spline = torch.where(r >= self.h / 2, t3, 2 * t3 - self.akinci_off)
            force = -p.surface_tension * ((spline / r)[:, None] * diff + nrm[i] - nrm[j])
            pull = self.total(i, (2 * p.rest_density / (rho[i] + rho[j]))[:, None] * force) * self.dt
        if swirl:
            v = v + torch.where((e2 > 1e-3)[:, None], turn, torch.zeros_like(turn))
        if tension:
            v = v + pull
        if viscous:
            i, j, d2 = full
            weigh = self.poly6(d2)
            if self.textbook:
                weigh = weigh * self.mass[j] / rho[j]
            v = v + p.xsph_c * self.total(i, weigh[:, None] * (v[j] - v[i]))
        return v
