"""The step's performance cases: what a program that simulates with this
framework has it do frame after frame, through JGS2GpuSolver, JGS2Batch and
JGS2Server.

Every pass is one turn of a host loop: upload what the host changed
(objectives), step one frame, read the pose and the velocities back.  A served
pass submits a few requests and waits for their results.

The scenes are the workloads of `jgs2_b200.scenes` and `bench.py`: cantilever
bars at 1-3x resolution, the unit cube, uneven batched bodies over a penalty
floor, the reference's one-cell IPC trough, the 8^3-hex box trough and the
cloth drape through the device broad phase, the contact-free sheet, and the
co-rotated bars of the demo scenes.  Rest meshes and their trained cubature are
fixed by a case's sizes (a program keeps them, or loads them from a fingerprinted
artifact); the pose, the velocities and the forces come from the seed.

`exact` runs the same frames in 64 bits with plain torch: the tetrahedral
paths (stable Neo-Hookean under both schedules, co-rotated linear, batches).
The cloth and IPC contact cases return None: their frames take decisions
(candidate activity, safe step, barrier line search) over up to millions of
candidates that a plain vectorised evaluation does not finish in 20 seconds.
"""
import dataclasses
import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "webgpu-physics_b200"))

from jgs2_b200 import scenes, server, solver  # noqa: E402

GGS2 = "graph-colored-gauss-seidel"
CUBE_EDGE = 100  # the headline cube: 1 030 301 vertices, 6 000 000 tets


def listed():
    return [
        # The smallest call of a per-frame loop: the minimal cantilever (525
        # vertices), 10 Jacobi iterations; launches and latency count.
        dict(name="bar_jacobi", kind="bar", nx=20, ny=4, nz=4, schedule="jacobi", iterations=10, young=1e5,
             forces=False),
        # The same bar under the graph-coloured schedule: about 20 colours an
        # iteration, each a few dozen vertices.
        dict(name="bar_coloured", kind="bar", nx=20, ny=4, nz=4, schedule=GGS2, iterations=6, young=1e5,
             forces=False),
        # An ordinary body of odd sizes that the host pushes: a new force
        # field every frame.
        dict(name="bar_forces", kind="bar", nx=61, ny=17, nz=11, schedule="jacobi", iterations=10, young=5e4,
             forces=True),
        # A mid-sized block under the graph-coloured schedule.
        dict(name="block_coloured", kind="bar", nx=37, ny=29, nz=23, schedule=GGS2, iterations=5, young=1e5,
             forces=False),
        # The co-rotated demo material with trained linear cubature.
        dict(name="corotated", kind="corotated", nx=24, ny=7, nz=5, schedule="jacobi", iterations=7, young=1e4),
        # The reference's IPC trough: ten one-cell boxes, static candidates.
        dict(name="trough", kind="trough", boxes=10, iterations=3),
        # Boxes of 8^3 hexes (exact complement, 192 records per vertex) falling
        # into the trough of plates, broad phase.
        dict(name="boxes", kind="boxes", boxes=6, cells=8, iterations=15),
        # The serving mix's sheet without contact.
        dict(name="sheet", kind="sheet", cells=127, iterations=5),
        # The sheet draping over a sphere with self-contact, broad phase.
        dict(name="drape", kind="drape", cells=127, iterations=5),
        # Many uneven bodies in one batch over the penalty floor.
        dict(name="batch", kind="batch", count=64, least=4, most=32, iterations=10),
        # Requests of mixed sizes through the server, from submit to result.
        dict(name="served", kind="served", requests=8, frames=30, iterations=10),
        # The headline: one large body.
        dict(name="cube", kind="cube", cells=CUBE_EDGE, iterations=20),
    ]


def _log(rng, low, high):
    """An integer spread over the logarithm of [low, high]."""
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    kind = rng.choice(["bar", "bar", "bar", "coloured", "corotated", "trough", "boxes", "sheet", "drape", "batch",
                       "served", "cube"])
    if kind in ("bar", "coloured", "corotated"):
        nx = _log(rng, 12, 64)
        ny, nz = (min(nx, _log(rng, 3, 32)) for _ in range(2))
        case = dict(kind="corotated" if kind == "corotated" else "bar", nx=nx, ny=ny, nz=nz, schedule="jacobi",
                    iterations=rng.randint(4, 12), young=round(10 ** rng.uniform(4.5, 6.0)))
        if kind == "coloured":
            case.update(schedule=GGS2, iterations=rng.randint(3, 7), forces=False)
        elif kind == "bar":
            case.update(forces=rng.random() < 0.5)
        else:
            # Soft demo materials: trained linear cubature diverges on stiff ones.
            case.update(young=round(10 ** rng.uniform(3.7, 4.1)), iterations=rng.randint(3, 7))
            if nx * ny * nz < 4000 and rng.random() < 0.3:
                case.update(schedule=GGS2, iterations=rng.randint(2, 4))
        return case
    if kind == "trough":
        return dict(kind=kind, boxes=rng.randint(4, 12), iterations=rng.choice([3, 5, 7]))
    if kind == "boxes":
        return dict(kind=kind, boxes=rng.randint(1, 6), cells=rng.randint(3, 8), iterations=rng.randint(7, 15))
    if kind == "sheet":
        return dict(kind=kind, cells=_log(rng, 15, 127), iterations=rng.choice([3, 5, 7, 9]))
    if kind == "drape":
        return dict(kind=kind, cells=_log(rng, 24, 127), iterations=rng.choice([3, 5]))
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 4, 64), least=4, most=rng.randint(9, 32), iterations=rng.randint(5, 12))
    if kind == "served":
        return dict(kind=kind, requests=rng.randint(3, 10), frames=_log(rng, 6, 30), iterations=rng.randint(5, 10))
    return dict(kind=kind, cells=_log(rng, 24, CUBE_EDGE - 1), iterations=rng.randint(10, 20))


# ---- scenes (a case's sizes alone; a few are kept for further preparations) ----


@functools.lru_cache(maxsize=12)
def _bar(nx, ny, nz, young, model):
    sc = scenes.Scene()
    m = sc.add_material(1000.0, young, 0.4, model)
    sc.add_cuboid((nx, ny, nz), (0.0, 0.0, 0.0), (0.05 * nx, 0.05 * ny, 0.05 * nz), m, 0, scenes.FACE_X_MIN)
    sc.precompute(timestep=1 / 60, cubature_k=6, method=scenes.PRECOMPUTE_PATCH, patch_radius=2)
    return sc.pack()


@functools.lru_cache(maxsize=1)
def _cube(cells):
    return scenes.unit_cube(cells=cells)


@functools.lru_cache(maxsize=2)
def _bodies(count, least, most):
    return scenes.batched_scenes(count=count, min_cells=least, max_cells=most)


@functools.lru_cache(maxsize=2)
def _trough(boxes):
    return scenes.trough(boxes=boxes)


@functools.lru_cache(maxsize=2)
def _boxes(boxes, cells):
    return scenes.box_trough(boxes=boxes, cells=cells)


@functools.lru_cache(maxsize=2)
def _sheet(cells):
    return scenes.cloth_sheet(cells=cells)


@functools.lru_cache(maxsize=2)
def _drape(cells):
    return scenes.cloth_sphere(cells=cells)


# ---- seeded states -----------------------------------------------------------------

BODY_SETTINGS = dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floorStiffness=0.0, parityMode=True)
FLOOR_SETTINGS = dict(timestep=1 / 60, gravity=(0.0, -9.81, 0.0), floorHeight=0.24, floorStiffness=20000.0,
                      parityMode=True)


def _rng(seed, salt=0):
    return np.random.default_rng([int(seed), salt])


def _moving(inp, rng, linear, spin, stretch=0.0):
    """The scene in a seeded state: a rigid velocity, each body about its own
    centre, and (stretch) a per-axis stretch U[1 - stretch, 1 + stretch] of
    the pose, in which its pinned vertices are held."""
    V = inp.vertex_count
    pos = inp.positions.reshape(V, 4).copy()
    rest = inp.vertex_rest.reshape(V, 4).copy()
    info = inp.vertex_info.reshape(V, 4)
    free = info[:, 2] == 0
    if stretch:
        s = rng.uniform(1.0 - stretch, 1.0 + stretch, 3).astype(np.float32)
        pos[:, :3] *= s
        rest[~free, :3] = pos[~free, :3]
    vel = np.zeros((V, 4), dtype=np.float32)
    for body in np.unique(info[free, 3]):
        at = free & (info[:, 3] == body)
        x = pos[at, :3] - pos[at, :3].mean(axis=0)
        vel[at, :3] = linear + rng.normal(0.0, 0.1, 3) + np.cross(rng.normal(0.0, spin, 3), x)
    return dataclasses.replace(inp, positions=pos.reshape(-1), vertex_rest=rest.reshape(-1),
                               velocities=vel.reshape(-1))


def _input(case, seed):
    """(scene input or inputs, settings) of a case."""
    rng = _rng(seed)
    kind = case["kind"]
    if kind == "bar":
        inp = _bar(case["nx"], case["ny"], case["nz"], case["young"], scenes.MATERIAL_STABLE_NEO_HOOKEAN)
        return _moving(inp, rng, 0.0, 0.3, 0.03), dict(BODY_SETTINGS, schedule=case["schedule"])
    if kind == "corotated":
        inp = _bar(case["nx"], case["ny"], case["nz"], case["young"], scenes.MATERIAL_COROTATED_LINEAR)
        return _moving(inp, rng, 0.0, 0.3), dict(BODY_SETTINGS, schedule=case["schedule"])
    if kind == "cube":
        return _moving(_cube(case["cells"]), rng, 0.0, 0.3, 0.03), dict(BODY_SETTINGS)
    if kind == "batch":
        parts = _bodies(case["count"], case["least"], case["most"])
        return [_moving(p, rng, np.array([0.0, -1.0, 0.0]), 0.3) for p in parts], dict(FLOOR_SETTINGS)
    if kind == "served":
        sizes = [1, 2, 1, 3, 1, 2, 1, 1, 2, 1][:case["requests"]]
        parts = [_bar(20 * r, 4 * r, 4 * r, 1e5, scenes.MATERIAL_STABLE_NEO_HOOKEAN) for r in sizes]
        return [_moving(p, rng, 0.0, 0.3, 0.03) for p in parts], dict(BODY_SETTINGS)
    if kind == "trough":
        return (_moving(_trough(case["boxes"]), rng, np.array([0.0, -3.0, 0.0]), 0.2),
                dict(scenes.TROUGH_SETTINGS, iterations=case["iterations"]))
    if kind == "boxes":
        return (_moving(_boxes(case["boxes"], case["cells"]), rng, np.array([0.0, -3.0, 0.0]), 0.2),
                dict(scenes.BOX_TROUGH_SETTINGS, iterations=case["iterations"]))
    inp = (_sheet if kind == "sheet" else _drape)(case["cells"])
    return _moving(inp, rng, 0.0, 0.05), dict(scenes.CLOTH_SETTINGS, iterations=case["iterations"])


def _force_fields(inp, seed):
    """Two smooth force fields, uploaded in turn (newtons per vertex)."""
    rng = _rng(seed, 1)
    x = inp.positions.reshape(-1, 4)[:, :3]
    free = inp.vertex_info.reshape(-1, 4)[:, 2:3] == 0
    mass = inp.vertex_rest.reshape(-1, 4)[:, 3:] * free
    return [(mass * (rng.normal(0.0, 3.0, 3) + np.sin(x @ rng.normal(0.0, 2.0, (3, 3))))).astype(np.float32)
            for _ in range(2)]


def prepare(case, seed):
    inputs, settings = _input(case, seed)
    kind = case["kind"]
    state = dict(kind=kind, iterations=case["iterations"], passes=0)
    if kind == "batch":
        state["batch"] = solver.JGS2Batch.create(inputs, settings)
        state["out"] = torch.empty(4 * sum(i.vertex_count for i in inputs), pin_memory=torch.cuda.is_available())
    elif kind == "served":
        state.update(server=server.JGS2Server(memoryBudgetBytes=16 << 30), inputs=inputs, settings=settings,
                     frames=case["frames"])
    else:
        state["solver"] = solver.JGS2GpuSolver.create(inputs, settings)
        state["out"] = torch.empty(4 * inputs.vertex_count, pin_memory=torch.cuda.is_available())
        if case.get("forces"):
            state["forces"] = _force_fields(inputs, seed)
    return state


def run(state):
    kind, n = state["kind"], state["iterations"]
    if kind == "served":
        ids = [state["server"].submit(i, state["settings"], frames=state["frames"], exactIterations=n)
               for i in state["inputs"]]
        done = [state["server"].wait(k) for k in ids]
        return dict(positions=[d["positions"] for d in done], velocities=[d["velocities"] for d in done])
    if kind == "batch":
        b = state["batch"]
        b.stepFrames(1, n)
        b.readAllPositions(state["out"].numpy())
        return dict(positions=state["out"], velocities=[b.readVelocities(i) for i in range(0, b.sceneCount, 8)])
    s = state["solver"]
    if "forces" in state:
        s.replaceExternalForces(state["forces"][state["passes"] % 2])
    state["passes"] += 1
    if kind in ("bar", "corotated", "cube", "boxes"):
        s.stepExactIterations(n)
    else:
        s.step()  # a production frame of the demo scenes (stop latch, odd iteration counts)
    s.readPositions(state["out"].numpy())
    return dict(positions=state["out"], velocities=s.readVelocities())


# ---- work ------------------------------------------------------------------------


def _counts(case):
    """(vertices, tets, records per vertex, cloth triangles, hinges) from the sizes alone."""
    kind = case["kind"]
    if kind in ("bar", "corotated"):
        n = (case["nx"], case["ny"], case["nz"])
        return (n[0] + 1) * (n[1] + 1) * (n[2] + 1), 6 * n[0] * n[1] * n[2], 6, 0, 0
    if kind == "cube":
        return (case["cells"] + 1) ** 3, 6 * case["cells"] ** 3, 6, 0, 0
    if kind == "batch":
        mean = (case["least"] + case["most"]) / 2
        return int(case["count"] * (mean + 1) ** 3), int(case["count"] * 6 * mean ** 3), 6, 0, 0
    if kind == "trough":
        return 12 + 8 * case["boxes"], 12 + 6 * case["boxes"], 6, 0, 0
    if kind == "boxes":
        c = case["cells"]
        return 340 + case["boxes"] * (c + 1) ** 3, 768 + case["boxes"] * 6 * c ** 3, 192, 0, 0
    c = case["cells"]
    extra = (8, 6) if kind == "sheet" else (729, 3072)
    return (c + 1) ** 2 + extra[0], extra[1], 4, 2 * c * c, 3 * c * c - 2 * c


def work(case):
    """Bytes: per iteration the state in and out of every vertex (source and
    target pose, inertial target, mass, connectivity, frame), each cubature
    record (id, weight, 36-float basis), each tetrahedron's record and
    incidence, each cloth triangle and hinge; per frame the prediction and the
    velocities.  Flops: the local systems and one line-search trial (about
    1 000 per record, 500 per incident tetrahedron and 300 per vertex, 1 000
    per cloth element), the assembled gate and the convergence gradient (300
    per tetrahedron and 400 per incidence)."""
    if case["kind"] == "served":
        total = {"bytes": 0, "flops": 0}
        for r in [1, 2, 1, 3, 1, 2, 1, 1, 2, 1][:case["requests"]]:
            one = work(dict(kind="bar", nx=20 * r, ny=4 * r, nz=4 * r, iterations=case["iterations"]))
            for k in total:
                total[k] += case["frames"] * one[k]
        return total
    V, T, K, C, H = _counts(case)
    n = case["iterations"]
    per = V * (84 + 152 * K) + 80 * T + 40 * C + 32 * H
    flops = 1000 * V * K + 900 * 4 * T + 300 * V + 300 * T + 1000 * (3 * C + 4 * H)
    return {"bytes": n * per + 64 * V, "flops": n * flops}


# ---- the same frames in 64 bits ----------------------------------------------------

UNIT, FLOOR_DET = 2.0 ** -24, float(np.float32(1e-4))


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _cof(f):
    a, b, c = f[..., 0], f[..., 1], f[..., 2]
    return torch.stack([_cross(b, c), _cross(c, a), _cross(a, b)], dim=-1)


def _dcof(f, h):
    a, b, c = f[..., 0], f[..., 1], f[..., 2]
    x, y, z = h[..., 0], h[..., 1], h[..., 2]
    return torch.stack([_cross(y, c) + _cross(b, z), _cross(z, a) + _cross(c, x), _cross(x, b) + _cross(a, y)], dim=-1)


def _det(f):
    return (f[..., 0] * _cross(f[..., 1], f[..., 2])).sum(-1)


def _unit(v, fallback):
    sq = (v * v).sum(-1, keepdim=True)
    return torch.where((sq > 1e-14) & (sq < 1e30), v / sq.clamp_min(1e-300).sqrt(), fallback)


def _polar(m):
    """Seven Newton steps towards the polar factor, then an orthonormal basis."""
    r = m
    done = torch.zeros(m.shape[0], dtype=torch.bool, device=m.device)
    for _ in range(7):
        d = _det(r)
        done = done | ~(d.abs() > 1e-7) | (d.abs() > 1e20)
        r = torch.where(done[:, None, None], r, 0.5 * (r + _cof(r) / torch.where(done, 1.0, d)[:, None, None]))
    ex, ey, ez = torch.eye(3, dtype=m.dtype, device=m.device).expand(m.shape[0], 3, 3).unbind(1)

    def beside(a):
        return _unit(_cross(a, torch.where(a[:, :1].abs() > 0.8, ey, ex)), ez)

    c0 = _unit(r[..., 0], ex)
    c1 = _unit(r[..., 1] - c0 * (c0 * r[..., 1]).sum(-1, keepdim=True), beside(c0))
    c2 = _unit(_cross(c0, c1), ez)
    flip = torch.where((c2 * r[..., 2]).sum(-1, keepdim=True) < 0, -1.0, 1.0)
    c2 = c2 * flip
    return torch.stack([c0, _unit(_cross(c2, c0), beside(c0)), c2], dim=-1)


class _Exact:
    """The step over concatenated tetrahedral scenes, every scene with its own
    accept / revert decision."""

    def __init__(self, inputs, settings, forces=None):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f64 = dict(dtype=torch.float64, device=dev)
        self.dev, self.f64 = dev, f64
        voff = np.cumsum([0] + [i.vertex_count for i in inputs])
        toff = np.cumsum([0] + [i.tet_count for i in inputs])
        K = self.K = inputs[0].cubature_k
        self.V, self.T, self.S = int(voff[-1]), int(toff[-1]), len(inputs)

        def cat(name, width, dtype=torch.float64):
            a = np.concatenate([getattr(i, name).reshape(-1, width) for i in inputs])
            return torch.from_numpy(a if dtype == torch.float64 else a.astype(np.int64)).to(dev, dtype)

        def shifted(name, width, off):
            a = [getattr(i, name).reshape(-1, width).astype(np.int64) + o for i, o in zip(inputs, off)]
            return torch.from_numpy(np.concatenate(a)).to(dev)

        self.x = cat("positions", 4)[:, :3].clone()
        self.vel = cat("velocities", 4)[:, :3].clone()
        rm = cat("vertex_rest", 4)
        self.rest, self.mass = rm[:, :3], rm[:, 3]
        info = cat("vertex_info", 4, torch.int64)
        self.n = info[:, 1].clamp_min(1).double()
        self.pinned = info[:, 2] != 0
        self.tets = shifted("tet_indices", 4, voff)
        dm = cat("tet_inverse_dm", 12).reshape(-1, 3, 4)  # three padded columns
        g = dm[:, :, :3].transpose(1, 2)                     # row l: the shape gradient of slot l + 1
        self.g = torch.cat([-g.sum(1, keepdim=True), g], dim=1)
        meta = cat("tet_meta", 4)
        self.vol, self.lam, self.mu = meta[:, 0], meta[:, 1], meta[:, 2]
        ids = np.concatenate([np.where(i.cubature_tet_ids < i.tet_count, i.cubature_tet_ids.astype(np.int64) + o, -1)
                              for i, o in zip(inputs, toff)])
        w = np.concatenate([i.cubature_weights for i in inputs]).astype(np.float64)
        at = np.flatnonzero((ids >= 0) & (w > 0))
        self.rt = torch.from_numpy(ids[at]).to(dev)
        self.rv = torch.from_numpy(at // K).to(dev)
        self.rw = torch.from_numpy(w[at]).to(dev)
        basis = np.concatenate([i.cubature_basis for i in inputs]).reshape(-1, 4, 3, 3)[at]
        self.ru = torch.from_numpy(basis).to(dev, torch.float64)
        self.own = (self.tets[self.rt] == self.rv[:, None]).double()  # the record's slot of its source vertex
        self.scene = torch.from_numpy(np.repeat(np.arange(self.S), np.diff(voff))).to(dev)
        self.tscene = torch.from_numpy(np.repeat(np.arange(self.S), np.diff(toff))).to(dev)
        self.stiff = None
        if inputs[0].tet_rest_stiffness is not None and float(meta[0, 3]) != 1.0:
            self.stiff = cat("tet_rest_stiffness", 144).reshape(-1, 12, 12)
        self.colors = None
        if settings.get("schedule") == GGS2:
            c = solver.build_vertex_coloring(inputs[0])[0]
            self.colors = torch.from_numpy(c.astype(np.int64)).to(dev)
        s = solver.resolve_settings(settings)
        f = np.float32
        self.dt = s["timestep"]
        self.ih2 = float(f((1.0 / self.dt) * (1.0 / self.dt)))
        self.gravity = torch.tensor(s["gravity"], **f64)
        self.maxStep, self.fh, self.fk, self.reg = s["max_step"], s["floor_height"], s["floor_stiffness"], s["regularization"]
        self.damping = s["velocity_damping"]
        scale = []
        for k in range(self.S):
            p = self.x[(self.scene == k) & ~self.pinned]
            scale.append((p.max(0).values - p.min(0).values).norm())
        self.scale = torch.stack(scale)[self.scene]
        self.force = torch.zeros(self.V, 3, **f64)
        if forces is not None:
            self.force = torch.from_numpy(forces).to(dev, torch.float64)

    def deform(self, x):
        return torch.einsum("tli,tlj->tij", x[self.tets], self.g)

    def gather(self, value):
        """Sum of per-slot values (T, 4, ...) over each vertex's incidences."""
        out = torch.zeros(self.V, *value.shape[2:], **self.f64)
        return out.index_add_(0, self.tets.reshape(-1), value.reshape(-1, *value.shape[2:]))

    def frames(self, F):
        vol = self.gather(self.vol[:, None].expand(-1, 4))
        avg = self.gather((self.vol[:, None, None] * F)[:, None].expand(-1, 4, 3, 3)) / vol.clamp_min(1e-300)[:, None, None]
        avg[vol <= 0] = torch.eye(3, **self.f64)
        return _polar(avg)

    def terms(self, F, lam, mu):
        i1 = (F * F).sum((-1, -2))
        cof, J = _cof(F), _det(F)
        a = mu * (1 - 1 / (i1 + 1))
        b = lam * (J - 1) - 0.75 * mu
        return cof, a, b, 2 * mu / (i1 + 1) ** 2

    def delta(self, F, D, lam, mu):
        """psi(F + D) - psi(F), without the cancellation of a difference, and det(F + D)."""
        f1 = F + D
        i0 = (F * F).sum((-1, -2))
        di = (D * (f1 + F)).sum((-1, -2))
        j0, j1 = _det(F), _det(f1)
        dj = (_cof(F) * D).sum((-1, -2)) + (_cof(D) * F).sum((-1, -2)) + _det(D)
        e = 0.5 * mu * di - 0.75 * mu * dj + 0.5 * lam * dj * (j1 + j0 - 2) - 0.5 * mu * torch.log1p(di / (i0 + 1))
        return e, j1

    def local(self, x, pred, todo):
        """The local solves of the vertices in `todo` at pose x: their new positions."""
        F = self.deform(x)
        R = self.frames(F)
        v_ok = todo & ~self.pinned
        keep = v_ok[self.rv]
        rv, rt, rw, own = self.rv[keep], self.rt[keep], self.rw[keep], self.own[keep]
        q = self.tets[rt]
        dW = torch.where(self.pinned, 0.0, self.mass * self.ih2 / self.n)
        share = torch.where(self.pinned, 0.0, 1.0 / self.n)
        B = torch.einsum("rlij,rljk,rmk->rlim", R[q], self.ru[keep], R[rv])
        lin = (dW[:, None] * (x - pred) - share[:, None] * self.force)
        gQ = torch.einsum("rlji,rlj->ri", B, lin[q])
        HQ = torch.einsum("rl,rlji,rljk->rik", dW[q], B, B)
        ownQ = own.sum(1) > 0
        inertia = self.mass * self.ih2
        grad = inertia[:, None] * (x - pred) - self.force
        hess = inertia[:, None, None] * torch.eye(3, **self.f64)
        low = (x[:, 1] < self.fh) & (self.fk > 0)
        grad[:, 1] += torch.where(low, self.fk * (x[:, 1] - self.fh), 0.0)
        hess[:, 1, 1] += torch.where(low, self.fk, 0.0)
        if self.stiff is not None:
            return self.corotated(x, F, B, rv, rt, rw, own, gQ, HQ, grad, hess, lin, dW, v_ok, ownQ)
        cof, a, b, c1 = self.terms(F, self.lam, self.mu)
        P = a[:, None, None] * F + b[:, None, None] * cof
        slotG = self.vol[:, None, None] * torch.einsum("tij,tlj->tli", P, self.g)
        u, w = torch.einsum("tij,tlj->tli", F, self.g), torch.einsum("tij,tlj->tli", cof, self.g)
        gg = (self.g * self.g).sum(-1)
        eye = torch.eye(3, **self.f64)
        slotH = self.vol[:, None, None, None] * (
            (a[:, None] * gg)[..., None, None] * eye + c1[:, None, None, None] * u[..., None] * u[..., None, :] +
            self.lam[:, None, None, None] * w[..., None] * w[..., None, :])
        grad = grad + self.gather(slotG)
        hess = hess + self.gather(slotH)
        # Cubature records: projected gradient and Hessian, less the source's own exact block.
        Fr, cr, ar, br, c1r = F[rt], cof[rt], a[rt], b[rt], c1[rt]
        lr, mr, vr = self.lam[rt], self.mu[rt], self.vol[rt]
        dF = torch.einsum("rlic,rlj->rcij", B, self.g[rt])
        pg = vr[:, None] * torch.einsum("rcij,rij->rc", dF, P[rt]) + gQ
        p, qq = torch.einsum("rcij,rij->rc", dF, Fr), torch.einsum("rcij,rij->rc", dF, cr)
        dc = torch.stack([_dcof(Fr, dF[:, c]) for c in range(3)], dim=1)
        ph = vr[:, None, None] * (ar[:, None, None] * torch.einsum("rcij,rdij->rcd", dF, dF) +
                                  c1r[:, None, None] * p[:, :, None] * p[:, None] +
                                  lr[:, None, None] * qq[:, :, None] * qq[:, None] +
                                  br[:, None, None] * torch.einsum("rcij,rdij->rcd", dF, dc)) + HQ
        pg = pg - torch.einsum("rl,rli->ri", own, slotG[rt]) - ownQ[:, None] * lin[rv]
        ph = ph - torch.einsum("rl,rlij->rij", own, slotH[rt]) - (ownQ * dW[rv])[:, None, None] * eye
        grad = grad.index_add(0, rv, rw[:, None] * pg)
        hess = hess.index_add(0, rv, rw[:, None, None] * ph)
        del ph, dc
        direction, ok = self.newton(hess, grad, inertia)
        return self.search(x, pred, F, dF, gQ, HQ, rv, rt, rw, own, ownQ, grad, inertia, direction, ok & v_ok, dW, share)

    def newton(self, hess, grad, inertia):
        h = 0.5 * (hess + hess.transpose(1, 2))
        diag = h.diagonal(dim1=1, dim2=2).abs().max(1).values
        scale = torch.maximum(inertia, torch.maximum(diag, ((h * h).sum((1, 2)) / 3).sqrt()))
        scale = torch.where(scale > 0, scale, 1.0)
        nh = h / scale[:, None, None]
        # Smallest eigenvalue in closed form.
        mean = nh.diagonal(dim1=1, dim2=2).sum(1) / 3
        d = nh - mean[:, None, None] * torch.eye(3, **self.f64)
        ss = ((d * d).sum((1, 2)) / 6).sqrt()
        half = (0.5 * _det(d / ss.clamp_min(1e-300)[:, None, None])).clamp(-1, 1)
        low = mean + 2 * ss * torch.cos(torch.acos(half) / 3 + 2 * np.pi / 3)
        shift = (2.0 ** -16 - low).clamp_min(0)
        m = nh + shift[:, None, None] * torch.eye(3, **self.f64)
        L, bad = torch.linalg.cholesky_ex(m)
        L = torch.where((bad == 0)[:, None, None], L, torch.eye(3, **self.f64))
        direction = torch.cholesky_solve((-grad / scale[:, None])[..., None], L)[..., 0]
        gd = (grad * direction).sum(1)
        ok = (shift <= float(np.float32(1e-3))) & (bad == 0) & (gd < 0) & torch.isfinite(direction).all(1)
        return torch.where(ok[:, None], direction, 0.0), ok

    def search(self, x, pred, F, dF, gQ, HQ, rv, rt, rw, own, ownQ, grad, inertia, direction, live, dW, share):
        def length(v):
            return v.norm(dim=1)

        resolution = torch.maximum(self.scale, x.abs().max(1).values) * UNIT * 8
        dl = length(direction)
        live = live & (dl > resolution)
        alpha = torch.where((self.maxStep > 0) & (dl > self.maxStep), self.maxStep / dl.clamp_min(1e-300), 1.0)
        out = x.clone()
        floor = self.minimum[self.scene]
        gs = torch.einsum("rl,rlj->rj", own, self.g[rt])
        live = live & (floor > FLOOR_DET)
        for _ in range(13):
            if not bool(live.any()):
                break
            td = alpha[:, None] * direction
            tl, gd = length(td), (grad * td).sum(1)
            long = (tl > self.maxStep * (1 + 1e-12)) if self.maxStep > 0 else torch.zeros_like(live)
            live = live & (long | ((tl > resolution) & (gd < 0)))
            try_now = live & ~long
            de = torch.zeros(self.V, **self.f64)
            jmin = floor.clone()
            step = td[self.tets]  # (T, 4, 3): each slot's own step
            for slot in range(4):
                e, j = self.delta(F, step[:, slot, :, None] * self.g[:, slot, None, :], self.lam, self.mu)
                de.index_add_(0, self.tets[:, slot], self.vol * e)
                jmin.scatter_reduce_(0, self.tets[:, slot], j, "amin")
            tr = td[rv]
            e, j = self.delta(F[rt], torch.einsum("rc,rcij->rij", tr, dF), self.lam[rt], self.mu[rt])
            comp = self.vol[rt] * e + (tr * gQ).sum(1) + 0.5 * torch.einsum("ri,rij,rj->r", tr, HQ, tr)
            e, _ = self.delta(F[rt], tr[:, :, None] * gs[:, None], self.lam[rt], self.mu[rt])
            mine = ((dW[:, None] * (x - pred) - share[:, None] * self.force) * td).sum(1) + 0.5 * dW * (td * td).sum(1)
            comp = comp - torch.where(ownQ, self.vol[rt] * e + mine[rv], 0.0)
            de.index_add_(0, rv, rw * comp)
            jmin.scatter_reduce_(0, rv, j, "amin")
            de += inertia * (((x - pred) * td).sum(1) + 0.5 * (td * td).sum(1)) - (self.force * td).sum(1)
            if self.fk > 0:
                i, f = (x[:, 1] - self.fh).clamp_max(0), (x[:, 1] + td[:, 1] - self.fh).clamp_max(0)
                de += 0.5 * self.fk * (f - i) * (f + i)
            good = try_now & (jmin > FLOOR_DET) & (de <= float(np.float32(1e-4)) * gd)
            out = torch.where(good[:, None], x + td, out)
            live = live & ~good
            alpha = 0.5 * alpha
        return out

    def corotated(self, x, F, B, rv, rt, rw, own, gQ, HQ, grad, hess, lin, dW, v_ok, ownQ):
        q = self.tets
        R = _polar(F)
        mean = lambda y: y - y.mean(1, keepdim=True)  # noqa: E731
        disp = torch.einsum("tji,tlj->tli", R, mean(x[q])) - mean(self.rest[q])
        K = self.stiff.reshape(-1, 4, 3, 4, 3)
        slotG = torch.einsum("tij,tajbk,tbk->tai", R, K, disp)
        KB = torch.einsum("tij,tajbk,tmk->taibm", R, K, R)  # world blocks
        slotH = torch.stack([KB[:, l, :, l] for l in range(4)], dim=1)
        grad = grad + self.gather(slotG)
        hess = hess + self.gather(slotH)
        pg = torch.einsum("rlji,rlj->ri", B, slotG[rt]) + gQ
        ph = torch.einsum("raic,raibj,rbjd->rcd", B, KB[rt], B) + HQ
        pg = pg - torch.einsum("rl,rli->ri", own, slotG[rt]) - ownQ[:, None] * lin[rv]
        ph = ph - torch.einsum("rl,rlij->rij", own, slotH[rt]) - (ownQ * dW[rv])[:, None, None] * torch.eye(3, **self.f64)
        grad = grad.index_add(0, rv, rw[:, None] * pg)
        hess = hess.index_add(0, rv, rw[:, None, None] * ph)
        ds = hess.diagonal(dim1=1, dim2=2).abs().max(1).values.clamp_min(1.0)
        shift = (self.reg * ds).clamp_min(1e-9)
        m = 0.5 * (hess + hess.transpose(1, 2))
        l00 = (m[:, 0, 0] + shift).maximum(shift).sqrt()
        l10, l20 = m[:, 1, 0] / l00, m[:, 2, 0] / l00
        l11 = (m[:, 1, 1] + shift - l10 * l10).maximum(shift).sqrt()
        l21 = (m[:, 2, 1] - l20 * l10) / l11
        l22 = (m[:, 2, 2] + shift - l20 * l20 - l21 * l21).maximum(shift).sqrt()
        y0 = -grad[:, 0] / l00
        y1 = (-grad[:, 1] - l10 * y0) / l11
        y2 = (-grad[:, 2] - l20 * y0 - l21 * y1) / l22
        x2 = y2 / l22
        x1 = (y1 - l21 * x2) / l11
        d = torch.stack([(y0 - l10 * x1 - l20 * x2) / l00, x1, x2], dim=1)
        n = d.norm(dim=1, keepdim=True)
        d = torch.where((n > self.maxStep) & (self.maxStep > 0), d * (self.maxStep / n.clamp_min(1e-300)), d)
        return torch.where(v_ok[:, None], x + d, x)

    def least(self, x):
        out = torch.full((self.S,), float("inf"), **self.f64)
        return out.scatter_reduce_(0, self.tscene, _det(self.deform(x)), "amin")

    def frame(self, iterations):
        old = self.x
        pred = old + self.dt * self.damping * self.vel + self.dt * self.dt * self.gravity
        pred = torch.where(self.pinned[:, None], self.rest, pred)
        source = old if self.stiff is None else pred
        self.minimum = self.least(source)
        everyone = torch.ones(self.V, dtype=torch.bool, device=self.dev)
        for _ in range(iterations):
            sets = [everyone] if self.colors is None else [self.colors == c for c in range(int(self.colors.max()) + 1)]
            x = source
            for todo in sets:
                x = torch.where((todo & self.pinned)[:, None], self.rest, self.local(x, pred, todo))
            if self.stiff is not None:
                source = x
                continue
            least = self.least(x)
            ok = (self.minimum > FLOOR_DET) & (least > FLOOR_DET)
            self.minimum = torch.where(ok, least, self.minimum)
            source = torch.where(ok[self.scene][:, None], x, source)
        self.x = torch.where(self.pinned[:, None], self.rest, source) if self.stiff is not None else source
        self.vel = torch.where(self.pinned[:, None], 0.0, (self.x - old) / self.dt)

    def answer(self):
        one = torch.ones(self.V, 1, **self.f64)
        return (torch.cat([self.x, one], 1).reshape(-1).cpu(), torch.cat([self.vel, 0 * one], 1).reshape(-1).cpu())


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("bar", "corotated", "cube", "batch", "served"):
        return None
    if kind == "bar" and case["schedule"] == GGS2 and case["nx"] * case["ny"] * case["nz"] > 30000:
        return None  # a sweep of about 20 colours over a large body takes longer than 20 seconds
    inputs, settings = _input(case, seed)
    inputs = inputs if isinstance(inputs, list) else [inputs]
    e = _Exact(inputs, settings, _force_fields(inputs[0], seed)[0] if case.get("forces") else None)
    for _ in range(case.get("frames", 1)):
        e.frame(case["iterations"])
    x, v = e.answer()
    sizes = [4 * i.vertex_count for i in inputs]
    if kind == "served":
        return dict(positions=list(x.split(sizes)), velocities=list(v.split(sizes)))
    if kind == "batch":
        return dict(positions=x, velocities=list(v.split(sizes))[::8])
    return dict(positions=x, velocities=v)
