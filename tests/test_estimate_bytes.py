"""What a request's memory estimate counts per IPC candidate is what an engine
allocates for it (include/jgs2_server.h admits requests by the estimate)."""
import numpy as np

from jgs2_b200 import scenes, server


def test_listed_candidates():
    # Two lists of indices (16), scene (4), state (96), flag (4) and column (4);
    # distances (8), previous entry (4); four entries of two keys and two
    # values; 256 histogram counts per 1 024 candidates (1).
    inp = scenes.cloth_drape(cells=8, prefold=False, contact=scenes.CONTACT_SURFACE)
    got = []
    for capacity in (1 << 20, 1 << 21):
        inp.contact_capacity = capacity
        got.append(server.estimate_device_bytes(inp))
    assert got[1] - got[0] == (1 << 20) * (2 * (16 + 4 + 96 + 4 + 4) + 8 + 4 + 64 + 1)


def test_static_candidates():
    # Indices, scene, state, distances, flag, incidence and active entries; a
    # range and a count per vertex.
    inp = scenes.trough(3, contact=scenes.CONTACT_STATIC)
    without = scenes.trough(3, contact=scenes.CONTACT_NONE)
    assert np.array_equal(inp.cubature_tet_ids, without.cubature_tet_ids)
    per = 16 + 4 + 96 + 8 + 4 + 16 + 16
    extra = server.estimate_device_bytes(inp) - server.estimate_device_bytes(without)
    assert extra == per * inp.contact_candidate_count + 12 * inp.vertex_count
