"""A colour's solve takes the item form up to 7 104 vertices and four lanes per
vertex past that: a scene swept alone and beside a filler whose colours are
larger must take the same steps, bit for bit, backtracked ones among them.
"""
import numpy as np
import pytest

from jgs2_b200 import scenes, solver

pytestmark = pytest.mark.gpu

SETTINGS = dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floorStiffness=0.0, parityMode=True,
                schedule="graph-colored-gauss-seidel")


def _bar(cells, K=6):
    sc = scenes.Scene()
    m = sc.add_material(1000.0, 5e4, 0.4)
    sc.add_cuboid(cells, (0.0, 0.0, 0.0), tuple(0.05 * c for c in cells), m, 0, scenes.FACE_X_MIN)
    sc.precompute(timestep=1 / 60, cubature_k=K, method=scenes.PRECOMPUTE_PATCH, patch_radius=1)
    return sc.pack()


@pytest.fixture(scope="module")
def filler():
    return _bar((41, 41, 41))  # 74 088 vertices, at most eight colours carry nearly all of them


def _state(batch):
    d = batch.readGlobalizationDiagnostics(0)
    local = np.delete(d["local"], 8, axis=1)  # all but the accepted trial's energy delta
    return [batch.readPositions(0), batch.readVelocities(0), local, d["history"]]


def _same(inp, settings, filler, frames, iterations):
    got = []
    for extra in ([], [filler]):
        batch = solver.JGS2Batch.create([inp] + extra, [settings] + [SETTINGS] * len(extra))
        batch.stepFrames(frames, iterations)
        got.append(_state(batch))
        batch.destroy()
    for alone, beside in zip(*got):
        np.testing.assert_array_equal(beside, alone)
    return got[0][3]


# Vertices of a shake of up to 12 mm; floor and objectives on the last.
@pytest.mark.parametrize("cells,K,shake,objectives", [((1, 1, 1), 4, 0.0, False), ((8, 1, 2), 6, 0.012, False),
                                                      ((12, 4, 4), 6, 0.012, False), ((6, 3, 3), 9, 0.0, False),
                                                      ((10, 4, 4), 6, 0.006, True)])
def test_both_forms_of_a_colour_take_the_same_steps(cells, K, shake, objectives, filler):
    inp = _bar(cells, K=K)
    rng = np.random.default_rng(4)
    free = inp.vertex_info.reshape(-1, 4)[:, 2] == 0
    p = inp.positions.reshape(-1, 4)
    p[free, :3] += rng.uniform(-shake, shake, (free.sum(), 3)).astype(np.float32)
    settings = dict(SETTINGS)
    if objectives:
        inp.external_forces = (rng.normal(0, 0.05, (inp.vertex_count, 3)) * free[:, None]).astype(np.float32).reshape(-1)
        inp.target_positions = (p[:, :3] + np.float32(0.02)).reshape(-1).copy()
        inp.target_stiffnesses = (200.0 * (rng.random(inp.vertex_count) < 0.3) * free).astype(np.float32)
        settings.update(floorStiffness=3000.0, floorHeight=0.06)
    _same(inp, settings, filler, 2, 3)


# The shaken cantilever whose vertices backtrack two and three times.
def test_backtracked_steps_are_the_same(filler):
    inp = scenes.cantilever(cells=(12, 4, 4), method=scenes.PRECOMPUTE_PATCH)
    rng = np.random.default_rng(4)
    p = inp.positions.reshape(-1, 4)
    free = inp.vertex_info.reshape(-1, 4)[:, 2] == 0
    p[free, :3] += rng.uniform(-0.012, 0.012, (free.sum(), 3)).astype(np.float32)
    assert _same(inp, SETTINGS, filler, 1, 2)[:, 28].max() >= 2
