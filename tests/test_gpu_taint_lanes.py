"""The lanes that share a particle agree on how it divides (needs a GPU): the mark
that decides it may change while they read it, so all take the first lane's answer.
Here every lane of a group looks at a mark of its own."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPO = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("lanes", [1, 4, 8])
def test_lanes_of_a_particle_agree(cuda_device, lanes):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = REPO / "tests" / "_build"
    out.mkdir(exist_ok=True)
    so = out / "libtaint_check.so"
    csrc = REPO / "position-based-fluids_gb300" / "csrc"
    if lanes == 1 or not so.exists():
        run = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false",
                              "-shared", "-Xcompiler", "-fPIC", "-I", str(REPO / "include"), "-I", str(csrc),
                              str(REPO / "tests" / "cuda" / "taint_check.cu"), "-o", str(so)], capture_output=True, text=True)
        assert run.returncode == 0, run.stderr[-3000:]
    check = ctypes.CDLL(str(so)).taint_check
    marks = np.random.default_rng(lanes).integers(0, 2, 64).astype(np.uint32)
    answers = np.full(64, 7, np.uint32)
    pointer = ctypes.POINTER(ctypes.c_uint32)
    assert check(lanes, marks.ctypes.data_as(pointer), answers.ctypes.data_as(pointer)) == 0
    assert np.array_equal(answers, np.repeat(marks[::lanes], lanes))
