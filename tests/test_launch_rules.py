"""Which kernel a launch takes and what it asks of the device, without a GPU:
the host code of libjgs2.so launches against a pretended CUDA runtime
(fake_cudart.cpp), which records kernels instead of running them and refuses
what a device would refuse.
"""
import os
import re
import subprocess

import pytest

from jgs2_b200 import _ffi

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "webgpu-physics_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def launch(tmp_path_factory):
    """Runs script lines; per answered line (accepted, kernel with its template
    arguments, device, grid, block, shared)."""
    exe = str(tmp_path_factory.mktemp("fake") / "fake_cudart")
    lib = os.path.abspath(_ffi.LIB_DIR)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(CUDA, "include"), "-I", CSRC,
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", exe, "-rdynamic", "-L", lib, "-ljgs2",
                    f"-Wl,-rpath,{lib}", "-Wl,--allow-shlib-undefined"], check=True)

    def run(*lines):
        out = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True).stdout
        answers = []
        for line in out.splitlines():
            if line == "declined":
                answers.append((False, "declined", ()))
                continue
            status, name, device, grid, block, shared = line.split()
            kernel = re.search(r"\d(solveItemsKernel|solveKernel|coloredSweepKernel|convergenceKernel|prologueKernel)",
                               name).group(1)
            args = re.match(r"I((?:L[a-z]\d+E)+)E", name.split(kernel, 1)[1]).group(1)
            kernel += "<" + ",".join(re.findall(r"L[a-z](\d+)E", args)) + ">"
            answers.append((status == "ok", kernel, (int(device), int(grid), int(block), int(shared))))
        return answers

    return run


# Twelve records a vertex take more shared memory than a kernel has without
# asking: solid, cloth and contact solves, coloured lists, both sweeps, and the
# item form, on the first device and on one after it.
def test_every_device_may_use_its_shared_memory(launch):
    calls = ["solve 50000 12 1 0 0 0 0", "solve 50000 12 1 1 0 0 0", "solve 200 12 0 0 100 1 0",
             "solve 9000 12 0 0 0 1 0", "solve 2000 66 1 0 0 0 0", "sweep 12 0", "sweep 12 1"]
    first = launch("device 0", *calls)
    both = launch("device 0", *calls, "device 1", *calls)
    assert all(ok for ok, _, _ in first) and len(first) == len(calls)
    assert max(where[3] for _, _, where in first) > 48 * 1024
    assert [(ok, kernel) for ok, kernel, _ in both] == 2 * [(ok, kernel) for ok, kernel, _ in first]
    assert [where[0] for _, _, where in both] == [0] * len(calls) + [1] * len(calls)


def _forms(answers):
    return [kernel for _, kernel, _ in answers]


# The item form's size rules are in waves of the device's own blocks.
@pytest.mark.parametrize("sms", [148, 100, 74])
def test_item_forms_follow_the_device(launch, sms):
    wave = 2 * sms
    script = [f"sms {sms}"]
    script += [f"solve {n} 6 1 0 0 0 0" for n in (1, 8 * wave, 8 * wave + 1, 16 * wave, 16 * wave + 1)]
    script += [f"solve {n} 6 0 0 0 1 0" for n in (1, 24 * wave, 24 * wave + 1)]
    assert _forms(launch(*script)) == [
        "solveItemsKernel<8,192,1,2>", "solveItemsKernel<8,192,1,2>", "solveItemsKernel<16,192,1,2>",
        "solveItemsKernel<16,192,1,2>", "solveItemsKernel<32,160,1,3>", "solveItemsKernel<8,192,0,2>",
        "solveItemsKernel<8,192,0,2>", "solveKernel<4,0,1>"]


# Eight lanes per vertex in the incident passes: solids up to 8 192 vertices,
# engines with cloth up to 28 672, the lanes' break-even there.
@pytest.mark.parametrize("kernel", ["convergence", "prologue"])
def test_the_incident_passes_change_form_where_both_measure_alike(launch, kernel):
    sizes = [(1, 0), (8192, 0), (8193, 0), (16392, 1), (28672, 1), (28673, 1), (32769, 1)]
    got = _forms(launch(*[f"{kernel} {v} {cloth}" for v, cloth in sizes]))
    assert got == [f"{kernel}Kernel<{wide}>" for wide in (1, 1, 0, 1, 1, 0, 0)]


# 32 vertices a block by item only where shared memory holds as many blocks as
# of four lanes, or one wave of them takes every vertex: not at 8 and 9 records
# past 9 472 vertices (148 SMs), nor at 12 to 14.
@pytest.mark.parametrize("vertices", [4737, 9472, 9473, 40000])
def test_wide_blocks_by_item_need_room(launch, vertices):
    widths = [1, 4, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 24, 40, 68]
    got = _forms(launch(*[f"solve {vertices} {k} 1 0 0 0 0" for k in widths]))
    lanes = {12, 13, 14} | ({8, 9} if vertices > 9472 else set())
    want = ["solveKernel<4,0,1>" if k in lanes else "solveItemsKernel<32,160,1,3>" for k in widths]
    assert got == want
    # The smaller forms take every width.
    for n, form in ((2368, 8), (4736, 16)):
        small = _forms(launch(*[f"solve {n} {k} 1 0 0 0 0" for k in widths]))
        assert small == [f"solveItemsKernel<{form},192,1,2>"] * len(widths)
