"""The contact passes where their rounds have remainders: rows of hundreds of
listed candidates (the carry window holds 64, a row's stored hit chunks 32),
vertices with more active candidates than a lane fetches ahead, and the
assembled gate on the caches a finished frame leaves.  A contact-surface run
must be its static run bit for bit.
"""
import numpy as np
import pytest

from jgs2_b200 import scenes, solver

pytestmark = pytest.mark.gpu


# Activation distances from a few listed pairs a row to nearly the superset
# (boxes of 0.46 m; 5^3 hexes give a row up to some 900 columns).
@pytest.mark.parametrize("cells", [2, 5])
@pytest.mark.parametrize("activation", [1e-3, 0.05, 0.3, 3.0])
def test_surface_run_is_the_static_run(cells, activation):
    args = dict(boxes=2, cells=cells, heights=(1.0, 1.3), plate_cells=(8, 2), method=scenes.PRECOMPUTE_PATCH,
                exact_complement=False, cubature_k=4)
    settings = dict(scenes.BOX_TROUGH_SETTINGS, ipcActivationDistance=activation, ipcBarrierStiffness=10.0)
    # Batches colour no scene: the static pile's conflict graph needs more
    # colours than the coloured schedule takes.
    a = solver.JGS2Batch.create([scenes.box_trough(contact=scenes.CONTACT_STATIC, **args)], settings)
    surface = scenes.box_trough(contact=scenes.CONTACT_SURFACE, **args)
    surface.contact_capacity = 1 << 22
    b = solver.JGS2Batch.create([surface], settings)
    for _ in range(3):
        a.stepFrames(1, 5)
        b.stepFrames(1, 5)
        np.testing.assert_array_equal(b.readPositions(0), a.readPositions(0))
        np.testing.assert_array_equal(b.readVelocities(0), a.readVelocities(0))
    np.testing.assert_array_equal(b.readGlobalizationDiagnostics(0)["local"],
                                  a.readGlobalizationDiagnostics(0)["local"])
    assert b.info(0)["contact_candidate_count"] > 0


# The gate after a frame reads the source caches that the accepted pose was
# promoted to, in static and listed form alike.
def test_gate_on_the_caches_of_a_finished_frame():
    out = []
    for contact in (scenes.CONTACT_STATIC, scenes.CONTACT_SURFACE):
        s = solver.JGS2GpuSolver.create(scenes.trough(3, contact=contact), scenes.TROUGH_SETTINGS)
        for _ in range(30):
            s.stepExactIterations(2)  # an even count leaves the list the gate reads by default in use
        pose = s.readPositions()
        r = s.evaluateAssembledCandidateForTest(pose, pose)
        out.append(r["control"])
        np.testing.assert_array_equal(r["positions"], pose)
    np.testing.assert_array_equal(out[0][:8], out[1][:8])
