"""Steps a bar with the checked library (JGS2_LIB_DIR) after lowering the
number of tets its index checks allow by one, alone and beside a filler, and
saves what each run read.  argv: output .npz, engine_view library.  Run by
tests/test_bounds_rejected.py."""
import ctypes
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "webgpu-physics_b200"))

import numpy as np  # noqa: E402

from jgs2_b200 import _ffi, scenes, solver  # noqa: E402

SETTINGS = dict(timestep=1 / 60, gravity=(0.0, -9.8, 0.0), floorStiffness=0.0, parityMode=True)


def bar(cells):
    sc = scenes.Scene()
    m = sc.add_material(1000.0, 5e4, 0.4)
    sc.add_cuboid(cells, (0.0, 0.0, 0.0), tuple(0.05 * c for c in cells), m, 0, scenes.FACE_X_MIN)
    sc.precompute(timestep=1 / 60, cubature_k=6, method=scenes.PRECOMPUTE_PATCH, patch_radius=1)
    return sc.pack()


def main(out, view):
    L = ctypes.CDLL(view)
    L.engine_tet_total.restype = ctypes.POINTER(ctypes.c_uint32)
    L.engine_tet_total.argtypes = [ctypes.c_void_p]
    inp = bar((12, 4, 4))
    saved = {}
    # Fillers past the item form's largest Jacobi engine and largest colour.
    for schedule, size in (("jacobi", 35), ("graph-colored-gauss-seidel", 41)):
        settings = dict(SETTINGS, schedule=schedule)
        for name, extra in (("items", []), ("lanes", [bar((size,) * 3)])):
            for rejected in (0, 1):
                batch = solver.JGS2Batch.create(extra + [inp], settings)
                total = L.engine_tet_total(batch._h)
                assert total[0] == sum(s.tet_count for s in extra + [inp])
                total[0] -= rejected  # the bar's last tet
                batch.stepFrames(1, 3)
                failed = False
                try:
                    batch.readVelocities(len(extra))  # the first read reports a failed check, once
                except _ffi.JGS2Error as e:
                    failed = "index check" in str(e)
                key = f"{schedule}/{name}/{rejected}/"
                saved[key + "failed"] = np.array([failed])
                saved[key + "positions"] = batch.readPositions(len(extra))
                saved[key + "local"] = batch.readGlobalizationDiagnostics(len(extra))["local"]
                batch.destroy()
    np.savez(out, **saved)


if __name__ == "__main__":
    main(sys.argv[1], sys.argv[2])
