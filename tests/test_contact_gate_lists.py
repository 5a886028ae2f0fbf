"""Which of a contact-surface engine's two candidate lists the calls after a
frame read: the list of the frame's last iteration, for odd and even iteration
counts, and again once an assembled-candidate evaluation has run.  The static
form of the scene has one list and says what the energies are.
"""
import numpy as np
import pytest

from jgs2_b200 import scenes, solver

pytestmark = pytest.mark.gpu


def _after_frames(contact, iterations, frames=60):
    s = solver.JGS2GpuSolver.create(scenes.trough(3, contact=contact), scenes.TROUGH_SETTINGS)
    for _ in range(frames):
        s.stepExactIterations(iterations)
    return s, s.readPositions()


def _pairs(candidates):
    return {tuple(int(i) for i in c) for c in np.asarray(candidates).reshape(-1, 4)}


# The energies are sums in double, folded in list order, of at most 4 200
# nonnegative terms and rounded to f32 once: two orders of the same terms agree
# to an f32 rounding (6e-8) and 4 200 double ones.
@pytest.mark.parametrize("iterations", [1, 2, 3, 4])
def test_the_gate_reads_the_last_list(iterations):
    stat, pose = _after_frames(scenes.CONTACT_STATIC, iterations)
    surf, surface_pose = _after_frames(scenes.CONTACT_SURFACE, iterations)
    np.testing.assert_array_equal(surface_pose, pose)
    want = stat.evaluateAssembledCandidateForTest(pose, pose)["control"]
    got = surf.evaluateAssembledCandidateForTest(pose, pose)["control"]
    np.testing.assert_array_equal(got[:8], want[:8])
    np.testing.assert_allclose(got[8:12], want[8:12], rtol=1.2e-7, atol=0)
    # The pose touches: without contact its energy is another.
    none = solver.JGS2GpuSolver.create(scenes.trough(3, contact=scenes.CONTACT_NONE), scenes.TROUGH_SETTINGS)
    free = none.evaluateAssembledCandidateForTest(pose, pose)["control"]
    assert want[9] > free[9] * (1 + 1e-4)
    # A second evaluation finds the same list.
    np.testing.assert_array_equal(surf.evaluateAssembledCandidateForTest(pose, pose)["control"], got)


# The listed pairs are those of the last iteration before and after an
# evaluation (which leaves one submitted iteration), not the other list's.
def test_the_listed_candidates_survive_an_evaluation():
    s, pose = _after_frames(scenes.CONTACT_SURFACE, 2, frames=40)
    before = _pairs(s.readContactCandidates())
    s.evaluateAssembledCandidateForTest(pose, pose)
    assert _pairs(s.readContactCandidates()) == before


# A frame without contact (barrier stiffness 0) lists nothing; the calls after
# it keep reading the last list there is.
def test_a_frame_without_contact_keeps_the_list():
    s, _ = _after_frames(scenes.CONTACT_SURFACE, 1, frames=40)
    before = _pairs(s.readContactCandidates())
    s.stepExactIterations(2, dict(ipcBarrierStiffness=0.0))
    assert _pairs(s.readContactCandidates()) == before
