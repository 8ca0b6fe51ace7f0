"""The counting sort of a bounds-checked build (needs a GPU): a key beyond the cell
table is reported by the kernels that look it up, and keys within it report
nothing.  The planted keys stay inside the test's own buffers."""
from __future__ import annotations

import ctypes
import os
import shutil
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPO = Path(__file__).resolve().parent.parent
CELL_KEY = 8  # kErrCellKey


@pytest.fixture(scope="module")
def check():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = REPO / "tests" / "_build"
    out.mkdir(exist_ok=True)
    so = out / "libchecked_sort.so"
    csrc = REPO / "position-based-fluids_gb300" / "csrc"
    run = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-DPBF_CHECK_BOUNDS",
                          "-shared", "-Xcompiler", "-fPIC", "-I", str(REPO / "include"), "-I", str(csrc),
                          str(REPO / "tests" / "cuda" / "checked_sort_check.cu"), str(csrc / "pbf_sort.cu"), "-o", str(so)],
                         capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-3000:]
    return ctypes.CDLL(str(so)).checked_sort


@pytest.mark.parametrize("beyond", [[], [0], [7, 999]])
def test_keys_beyond_the_table_are_reported(check, cuda_device, beyond):
    n, limit = 1000, 64
    keys = np.random.default_rng(3).integers(0, limit, n).astype(np.uint32)
    keys[beyond] = limit + 1 + np.arange(len(beyond))
    place = np.zeros(n, np.uint32)
    for k in np.unique(keys):
        place[keys == k] = np.arange((keys == k).sum())
    errors = (ctypes.c_int * 2)(-1, -1)
    pointer = ctypes.POINTER(ctypes.c_uint32)
    assert check(n, ctypes.c_uint32(limit), keys.ctypes.data_as(pointer), place.ctypes.data_as(pointer), errors) == 0
    for word in errors:
        assert bool(word & CELL_KEY) == bool(beyond)
        assert beyond or word == 0


RENDER = """
import sys
sys.path[:0] = [{repo!r}, {pkg!r}]
import numpy as np
import pbf
from oracle import oracle
assert pbf.LIB_PATH.name == "libpbf_gb300_checked.so", pbf.LIB_PATH
params = pbf.load_scenario("dam_break_32k")
params.h, params.h_2 = 2.0, 4.0
pos = pbf.scene_block(16, 16, 16, 0.55, (0.3, 0.3, 0.3), 0.05, 7)
params.particleCount = len(pos)
cam = pbf.render_camera((4.4, 8.0, 30.0), (4.4, 4.0, 4.4), (0.0, 1.0, 0.0), 45.0, 320, 240, 1.0)
with pbf.Simulation.create(params, pos, np.zeros_like(pos), device=0) as sim:
    sim.render_frame(cam, 0)
    out = sim.render_read(cam, 0)
    sim.synchronize()  # raises if a kernel reported an index out of range
want = oracle.render(cam, 0, params, pos)[2]
a, b = (np.where(np.isnan(x), np.float32(7), x) for x in (out, want))
assert np.array_equal(a, b)
print("checked render ok")
"""


def test_checked_render_reports_nothing(cuda_device):
    build = REPO / "position-based-fluids_gb300" / "build.py"
    run = subprocess.run([sys.executable, str(build), "--checked"], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stderr[-3000:]
    run = subprocess.run([sys.executable, "-c", RENDER.format(repo=str(REPO), pkg=str(REPO / "position-based-fluids_gb300"))],
                         env=dict(os.environ, PBF_CHECK_BOUNDS="1"), capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout[-3000:] + run.stderr[-3000:]
    assert "checked render ok" in run.stdout
