"""What a checked build's solve does with an incident tet that its index check
rejects: the tet's terms are left out, in the item form as with four lanes per
vertex, and the first read after the frame fails.  The check is made to
reject by lowering the limit it holds the index against; the tet's data is
there, so nothing is read out of range whatever the kernel does.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CHECKED = os.environ.get("JGS2_CHECKED_DIR") or os.path.join(ROOT, "webgpu-physics_b200", "lib", "checked")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("rejected")
    view, out = str(tmp / "engine_view.so"), str(tmp / "runs.npz")
    subprocess.run(["g++", "-std=c++17", "-O0", "-w", "-shared", "-fPIC", "-DJGS2_BOUNDS_CHECKS=1",
                    "-I", os.path.join(CUDA, "include"), "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "webgpu-physics_b200", "csrc"), os.path.join(HERE, "engine_view.cpp"),
                    "-o", view, "-L", CHECKED, "-ljgs2", f"-Wl,-rpath,{CHECKED}", "-Wl,--allow-shlib-undefined"],
                   check=True)
    res = subprocess.run([sys.executable, os.path.join(HERE, "rejected_run.py"), out, view],
                         env=dict(os.environ, JGS2_LIB_DIR=CHECKED), capture_output=True, text=True, timeout=900)
    assert res.returncode == 0, res.stderr[-3000:]
    return np.load(out)


@pytest.mark.parametrize("schedule", ["jacobi", "graph-colored-gauss-seidel"])
def test_a_rejected_tet_is_left_out_by_every_form(schedule, runs):
    def read(name, rejected, key):
        return runs[f"{schedule}/{name}/{rejected}/{key}"]

    for name in ("items", "lanes"):
        assert not read(name, 0, "failed")[0] and read(name, 1, "failed")[0]
        assert not np.array_equal(read(name, 0, "positions"), read(name, 1, "positions"))
    # Both forms take the same steps with every tet and without the rejected one
    # (local records but for the accepted trial's energy delta).
    for rejected in (0, 1):
        np.testing.assert_array_equal(read("items", rejected, "positions"), read("lanes", rejected, "positions"))
        items, lanes = (np.delete(read(n, rejected, "local"), 8, axis=1) for n in ("items", "lanes"))
        np.testing.assert_array_equal(items, lanes)
