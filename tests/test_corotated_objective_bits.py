"""A co-rotated record takes the vertex's own objective share out of its
gradient with one fused multiply-add.  The expected update lengths (f32 words)
of one vertex of a one-hex cube under forces and target springs are those of
the one-thread-per-vertex solve that the solve by items replaced; with the
share rounded before it is taken out each differs in its last bits.
"""
import numpy as np
import pytest

from jgs2_b200 import scenes, solver

pytestmark = pytest.mark.gpu

EXPECTED = {6: 0x3c7b1c5c, 12: 0x3c88f7a0, 24: 0x3cd0073d, 33: 0x3c5d948c, 99: 0x3c718251, 152: 0x3c700b8b,
            163: 0x3bdfef18, 208: 0x3c38fb74, 217: 0x3ba17e78, 250: 0x3c4a2655}


@pytest.fixture(scope="module")
def cube():
    sc = scenes.Scene()
    m = sc.add_material(1000.0, 1e4, 0.3, scenes.MATERIAL_COROTATED_LINEAR)
    sc.add_cuboid((1, 1, 1), (0.0, 0.0, 0.0), (0.05, 0.05, 0.05), m, 0, scenes.FACE_X_MIN)
    sc.precompute(timestep=1 / 60, cubature_k=6, method=scenes.PRECOMPUTE_PATCH, patch_radius=1)
    return sc.pack()


@pytest.mark.parametrize("seed", sorted(EXPECTED))
def test_own_objective_share_is_fused(seed, cube):
    rng = np.random.default_rng(seed)
    inp = cube.copy()
    V = inp.vertex_count
    free = inp.vertex_info.reshape(-1, 4)[:, 2] == 0
    inp.external_forces = (rng.normal(0, 0.05, (V, 3)) * free[:, None]).astype(np.float32).reshape(-1)
    offset = rng.normal(0, 0.02, (V, 3)).astype(np.float32)
    inp.target_positions = (inp.positions.reshape(-1, 4)[:, :3] + offset).reshape(-1).copy()
    inp.target_stiffnesses = (200.0 * (rng.random(V) < 0.6) * free).astype(np.float32)
    s = solver.JGS2GpuSolver.create(inp, dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floorStiffness=0.0,
                                              parityMode=True))
    s.stepExactIterations(1)
    assert int(s.readFinalIterationUpdates()[28:29].view(np.uint32)[0]) == EXPECTED[seed]  # vertex 7
