"""The local solve of solid scenes picks its form by the number of vertices it
solves: blocks of 8, 16 or 32 vertices by item, or four lanes per vertex.  All
forms take the same steps, so a scene must give the same bits alone and beside
fillers that push the engine into the next form, with and without the terms a
vertex can carry; and a sweep with more incident tets or records than one
round takes must follow the oracle (positions within 1e-4 of the bounding-box
diagonal, accept flags equal).
"""
import math

import numpy as np
import pytest

from jgs2_b200 import scenes, solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SETTINGS = dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floorStiffness=0.0, parityMode=True)
GGS2 = "graph-colored-gauss-seidel"


def _bar(cells, young=5e4, K=6, origin=(0.0, 0.0, 0.0), exact=False):
    sc = scenes.Scene()
    m = sc.add_material(1000.0, young, 0.4)
    sc.add_cuboid(cells, origin, tuple(0.05 * c for c in cells), m, 0, scenes.FACE_X_MIN)
    sc.precompute(timestep=1 / 60, cubature_k=K, method=scenes.PRECOMPUTE_PATCH, patch_radius=1,
                  exact_complement=1 if exact else 0)
    return sc.pack()


@pytest.fixture(scope="module")
def fillers():
    """(vertices, scene): with a small scene, 16, 32 and 4 lanes per vertex."""
    return [_bar((24, 10, 9)), _bar((20, 20, 19)), _bar((34, 34, 34))]  # 2 750, 8 820, 42 875 vertices


def _state(batch, i):
    d = batch.readGlobalizationDiagnostics(i)
    local = np.delete(d["local"], 8, axis=1)  # all but the accepted trial's energy delta
    return [batch.readPositions(i), batch.readVelocities(i), local, d["history"]]


# 8 vertices (one block), 9 and 15 more than whole blocks of 8, 16 and 32;
# floor and objectives on the last.
@pytest.mark.parametrize("cells,K,objectives", [((1, 1, 1), 4, False), ((8, 1, 2), 6, False), ((6, 3, 3), 9, False),
                                                ((10, 4, 4), 6, True)])
def test_every_form_takes_the_same_steps(cells, K, objectives, fillers):
    inp = _bar(cells, K=K)
    settings = dict(SETTINGS)
    if objectives:
        rng = np.random.default_rng(3)
        free = inp.vertex_info.reshape(-1, 4)[:, 2] == 0
        inp.external_forces = (rng.normal(0, 0.05, (inp.vertex_count, 3)) * free[:, None]).astype(np.float32).reshape(-1)
        inp.target_positions = (inp.positions.reshape(-1, 4)[:, :3] + np.float32(0.02)).reshape(-1).copy()
        inp.target_stiffnesses = (200.0 * (rng.random(inp.vertex_count) < 0.3) * free).astype(np.float32)
        settings.update(floorStiffness=3000.0, floorHeight=0.06)
    want = None
    for extra in [[]] + [[f] for f in fillers]:
        batch = solver.JGS2Batch.create([inp] + extra, [settings] + [SETTINGS] * len(extra))
        for _ in range(2):
            batch.stepFrames(1, 4)
        got = _state(batch, 0)
        batch.destroy()
        want = want or got
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b)


# A stiff cube whose vertices backtrack past the first trial: by items the later
# trials are evaluated four at a time, by lanes one by one.
def test_backtracked_trials_are_judged_in_order(fillers):
    inp = scenes.unit_cube(cells=6)
    want = None
    for extra in [[]] + [[f] for f in fillers]:
        batch = solver.JGS2Batch.create([inp] + extra, SETTINGS)
        batch.stepFrames(1, 4)
        got = _state(batch, 0)
        batch.destroy()
        want = want or got
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b)
    assert want[3][:, 28].max() >= 1  # some vertex went past its first trial


def _against_oracle(inp, schedule, iterations):
    s = dict(SETTINGS, schedule=schedule)
    g = solver.JGS2GpuSolver.create(inp, s)
    c = O.OracleSolver(inp, dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floor_stiffness=0.0, parity_mode=1,
                                 schedule=solver.SCHEDULES[schedule]))
    g.stepExactIterations(iterations)
    c.step_exact_iterations(iterations)
    a = g.readPositions().reshape(-1, 4)[:, :3].astype(np.float64)
    b = c.read("positions").reshape(-1, 4)[:, :3].astype(np.float64)
    assert np.abs(a - b).max() <= 1e-4 * inp.bbox_diagonal()
    hg = g.readGlobalizationDiagnostics()
    hc = np.asarray(c.read("history"), dtype=np.float32).reshape(-1, 32)[:iterations]
    np.testing.assert_array_equal(hg["history"][:, 4:6], hc[:, 4:6])
    return hg["history"]


def _fan(n):
    """n tets around one edge: its two vertices have n incident tets each."""
    ring = [(0.2 * math.cos(2 * math.pi * i / n), 0.0, 0.2 * math.sin(2 * math.pi * i / n)) for i in range(n)]
    pos = np.array([(0.0, -0.1, 0.0), (0.0, 0.1, 0.0)] + ring)
    tets = np.array([[0, 1, 2 + (i + 1) % n, 2 + i] for i in range(n)])
    p = pos[tets[0]]
    if np.linalg.det(p[1:] - p[0]) < 0:
        tets[:, 2:] = tets[:, :1:-1].copy()
    pinned = np.zeros(n + 2, dtype=np.uint8)
    pinned[2] = pinned[2 + n // 2] = 1
    sc = scenes.Scene()
    m = sc.add_material(1000.0, 1e4, 0.3)
    sc.add_mesh(pos.reshape(-1), tets.reshape(-1), m, pinned=pinned)
    sc.precompute(timestep=1 / 60, cubature_k=n, exact_complement=1)
    return sc.pack()


@pytest.mark.parametrize("schedule", ["jacobi", GGS2])
@pytest.mark.parametrize("n", [24, 25, 49])
def test_more_incident_tets_than_a_round(n, schedule):
    _against_oracle(_fan(n), schedule, 2)


# The widest cached records (K <= 68 at 240 bytes each) leave a block fewer vertices.
@pytest.mark.parametrize("schedule", ["jacobi", GGS2])
def test_wide_cached_records(schedule):
    _against_oracle(_bar((2, 1, 1), K=60, exact=True), schedule, 2)


# A bar shaken until vertices backtrack two and three times (seeded): the f32
# and FP64 oracles agree on it to 3e-7 of the diagonal.
@pytest.mark.parametrize("schedule", ["jacobi", GGS2])
def test_backtracking_follows_the_oracle(schedule):
    inp = scenes.cantilever(cells=(12, 4, 4), method=scenes.PRECOMPUTE_PATCH)
    rng = np.random.default_rng(4)
    p = inp.positions.reshape(-1, 4)
    free = inp.vertex_info.reshape(-1, 4)[:, 2] == 0
    p[free, :3] += rng.uniform(-0.012, 0.012, (free.sum(), 3)).astype(np.float32)
    assert _against_oracle(inp, schedule, 2)[:, 28].max() >= 2
