"""The co-rotated solve takes ten vertices a block, 24 incident tets and 8
records of a vertex per round: frames against the oracle where those rounds
and blocks have remainders, with every term a vertex can carry.  Positions
within 1e-4 of the bounding-box diagonal, as in the other parity tests.
"""
import math

import numpy as np
import pytest

from jgs2_b200 import scenes, solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-4
COROTATED = scenes.MATERIAL_COROTATED_LINEAR


def _bar(cells, K, exact):
    sc = scenes.Scene()
    m = sc.add_material(1000.0, 1e4, 0.3, COROTATED)
    sc.add_cuboid(cells, (0.0, 0.0, 0.0), tuple(0.05 * c for c in cells), m, 0, scenes.FACE_X_MIN)
    args = dict(timestep=1 / 60, cubature_k=K, method=scenes.PRECOMPUTE_PATCH, patch_radius=1)
    sc.precompute(exact_complement=1 if exact else 0, **args)
    return sc.pack()


def _fan(n):
    """n tets around one edge: its two vertices have n incident tets each."""
    ring = [(0.2 * math.cos(2 * math.pi * i / n), 0.0, 0.2 * math.sin(2 * math.pi * i / n)) for i in range(n)]
    tets = []
    for i in range(n):
        tets += [0, 1, 2 + (i + 1) % n, 2 + i]
    sc = scenes.Scene()
    m = sc.add_material(1000.0, 1e4, 0.3, COROTATED)
    pos = np.array([(0.0, -0.1, 0.0), (0.0, 0.1, 0.0)] + ring)
    p = pos[np.array(tets[:4])]
    if np.linalg.det(p[1:] - p[0]) < 0:
        tets = [t for q in np.array(tets).reshape(-1, 4) for t in (q[0], q[1], q[3], q[2])]
    pinned = np.zeros(n + 2, dtype=np.uint8)
    pinned[2] = pinned[2 + n // 2] = 1
    sc.add_mesh(pos.reshape(-1), tets, m, pinned=pinned)
    sc.precompute(timestep=1 / 60, cubature_k=n, exact_complement=1)
    return sc.pack()


def _compare(inp, settings, schedule, iterations, objectives):
    s = dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), parityMode=True, schedule=schedule, **settings)
    g = solver.JGS2GpuSolver.create(inp, s)
    o = {solver.CAMEL.get(k, k): v for k, v in s.items()}
    o.update(parity_mode=1, schedule=solver.SCHEDULES[schedule])
    c = O.OracleSolver(inp, o)
    if objectives:
        rng = np.random.default_rng(5)
        free = inp.vertex_info.reshape(-1, 4)[:, 2] == 0
        f = (rng.normal(0.0, 0.01, (inp.vertex_count, 3)) * free[:, None]).astype(np.float32)
        t = inp.positions.reshape(-1, 4)[:, :3] + np.float32(0.01)
        k = (50.0 * (rng.random(inp.vertex_count) < 0.3) * free).astype(np.float32)
        g.replaceExternalForces(f)
        g.replaceQuadraticTargets(t, k)
        c.set_objectives(f.reshape(-1), np.ascontiguousarray(t).reshape(-1), k)
    g.stepExactIterations(iterations)
    c.step_exact_iterations(iterations)
    a = g.readPositions().reshape(-1, 4)[:, :3].astype(np.float64)
    b = c.read("positions").reshape(-1, 4)[:, :3].astype(np.float64)
    assert np.isfinite(a).all()
    assert np.abs(a - b).max() <= TOL * inp.bbox_diagonal()


# 8 vertices (less than a block), 20 and 24 (two full blocks, a remainder);
# 1, 8 and 9 records (one, a full round, a second round) and every candidate.
@pytest.mark.parametrize("schedule", ["jacobi", "graph-colored-gauss-seidel"])
@pytest.mark.parametrize("cells,K,exact", [((1, 1, 1), 4, False), ((4, 1, 1), 1, False), ((5, 1, 1), 8, False),
                                           ((3, 2, 2), 9, False), ((3, 2, 2), 192, True)])
def test_rounds_and_blocks(cells, K, exact, schedule):
    _compare(_bar(cells, K, exact), dict(floorStiffness=0.0), schedule, 2, False)


@pytest.mark.parametrize("n", [24, 25, 49])
def test_more_incident_tets_than_a_round(n):
    _compare(_fan(n), dict(floorStiffness=0.0), "jacobi", 2, False)


def test_objectives_and_floor():
    _compare(_bar((6, 2, 2), 6, False), dict(floorStiffness=2000.0, floorHeight=0.04), "jacobi", 2, True)
