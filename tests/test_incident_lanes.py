"""The prologue and convergence passes sum a vertex's incident tets with eight
lanes in small engines and one thread in large ones, in entries of 32 vertices
that are folded in groups of 32.  Both forms add the same terms in the same
order, so a scene must give the same bits alone (eight lanes) and beside a
filler that makes the engine large (one thread), at vertex counts around the
entry and group edges; and its frame must stay within the parity bounds of the
oracle (positions within 1e-4 of the bounding-box diagonal, residuals 5 %).
"""
import numpy as np
import pytest

from jgs2_b200 import scenes, solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SETTINGS = dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floorStiffness=0.0, parityMode=True)


def _bar(cells, pinned=scenes.FACE_X_MIN):
    sc = scenes.Scene()
    m = sc.add_material(1000.0, 5e4, 0.4)
    sc.add_cuboid(cells, (0.0, 0.0, 0.0), tuple(0.05 * c for c in cells), m, 0, pinned)
    sc.precompute(timestep=1 / 60, cubature_k=6, method=scenes.PRECOMPUTE_PATCH)
    return sc.pack()


@pytest.fixture(scope="module")
def filler():
    return _bar((20, 20, 20))  # 9 261 vertices: above the eight-lane limit of 8 192


# 8, 32 and 36 vertices (one entry, one full entry, a remainder of four), 1 024
# (one full group), 1 088 (two groups), 8 064 (the last grid below the limit).
@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 1, 1), (8, 1, 1), (15, 3, 15), (16, 3, 15), (27, 17, 15)])
def test_same_bits_in_both_forms(cells, filler):
    inp = _bar(cells)
    alone = solver.JGS2GpuSolver.create(inp, SETTINGS)
    both = solver.JGS2Batch.create([inp, filler], SETTINGS)
    for _ in range(2):
        alone.stepExactIterations(5)
        both.stepFrames(1, 5)
    np.testing.assert_array_equal(alone.readPositions(), both.readPositions(0))
    np.testing.assert_array_equal(alone.readVelocities(), both.readVelocities(0))
    a, b = alone.readGlobalizationDiagnostics(), both.readGlobalizationDiagnostics(0)
    np.testing.assert_array_equal(a["local"], b["local"])
    np.testing.assert_array_equal(a["history"], b["history"])


# Cloth elements are added by the same lanes, in engines of up to 40 000
# vertices: sheets of 33 and 1 164 vertices (with their collider's 8).
@pytest.mark.parametrize("cells", [4, 33])
def test_cloth_gives_the_same_bits_in_both_forms(cells):
    inp = scenes.cloth_sheet(cells=cells)
    settings = dict(scenes.CLOTH_SETTINGS)
    alone = solver.JGS2GpuSolver.create(inp, settings)
    both = solver.JGS2Batch.create([inp, _bar((34, 34, 34))], [settings, dict(SETTINGS, timestep=1 / 60)])
    for _ in range(3):
        alone.stepExactIterations(4)
        both.stepFrames(1, 4)
    np.testing.assert_array_equal(alone.readPositions(), both.readPositions(0))
    np.testing.assert_array_equal(alone.readVelocities(), both.readVelocities(0))
    a, b = alone.readGlobalizationDiagnostics(), both.readGlobalizationDiagnostics(0)
    np.testing.assert_array_equal(a["local"], b["local"])
    np.testing.assert_array_equal(a["history"], b["history"])


@pytest.mark.parametrize("cells", [(7, 1, 1), (16, 3, 15), (20, 20, 20)])
def test_frame_against_the_oracle(cells):
    inp = _bar(cells)
    gpu = solver.JGS2GpuSolver.create(inp, SETTINGS)
    cpu = O.OracleSolver(inp, dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floor_stiffness=0.0, parity_mode=1))
    gpu.stepExactIterations(5)
    cpu.step_exact_iterations(5)
    g = gpu.readPositions().reshape(-1, 4)[:, :3].astype(np.float64)
    c = cpu.read("positions").reshape(-1, 4)[:, :3].astype(np.float64)
    assert np.abs(g - c).max() <= 1e-4 * inp.bbox_diagonal()
    hg = gpu.readGlobalizationDiagnostics()["history"][:5]
    hc = np.asarray(cpu.read("history"), dtype=np.float32).reshape(-1, 32)[:5]
    np.testing.assert_array_equal(hg[:, 4:6], hc[:, 4:6])  # accept / revert
    np.testing.assert_allclose(hg[:, 17], hc[:, 17], rtol=5e-2)  # residual norm
