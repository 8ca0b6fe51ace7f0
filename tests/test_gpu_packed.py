"""The passes' packed arithmetic (two friends per instruction, csrc/
pbf_device.cuh) against its scalar form, bit for bit (needs a GPU): |r| and its
reciprocal on every float r^2 in [2^-100, 2^64), and the chain of r^2, quotients
and their squared sum on seeded differences.  Both forms are defined as the same
IEEE operations in the same order, so no mismatch is tolerated."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPO = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def lib():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = REPO / "tests" / "_build"
    out.mkdir(exist_ok=True)
    so = out / "libpacked_check.so"
    csrc = REPO / "position-based-fluids_gb300" / "csrc"
    run = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false",
                          "-shared", "-Xcompiler", "-fPIC", "-I", str(REPO / "include"), "-I", str(csrc),
                          str(REPO / "tests" / "cuda" / "packed_check.cu"), "-o", str(so)],
                         capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-3000:]
    lib = ctypes.CDLL(str(so))
    lib.packed_sqrt_check.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.POINTER(ctypes.c_ulonglong)]
    lib.packed_chain_check.argtypes = [ctypes.c_float, ctypes.c_uint32, ctypes.c_int,
                                       ctypes.POINTER(ctypes.c_ulonglong)]
    return lib


def test_square_root_and_reciprocal_equal_the_scalar_form(lib, cuda_device):
    lo, hi = (int(np.array(x, np.float32).view(np.uint32)) for x in (2.0 ** -100, 2.0 ** 64))
    bad = ctypes.c_ulonglong(1)
    assert lib.packed_sqrt_check(lo, hi, ctypes.byref(bad)) == 0
    assert bad.value == 0


@pytest.mark.parametrize("h2", [0.01, 0.0225, 4.0])
def test_chain_equals_the_scalar_form(lib, cuda_device, h2):
    bad = ctypes.c_ulonglong(1)
    assert lib.packed_chain_check(h2, 12345, 512, ctypes.byref(bad)) == 0
    assert bad.value == 0
