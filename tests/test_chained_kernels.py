"""Kernels that may start before the kernel ahead of them on the stream has ended
(launch_chained) and wait for its end themselves (chain_wait).  CPU: the sources
are read.  What the compiler may move ahead of the wait must not be there: each
such kernel waits in its first statement, and neither it nor anything in the files
that the chain's kernels share declares memory as unchanging while the kernel runs
(__restrict__, __ldg, ld.global.nc)."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "position-based-fluids_gb300" / "csrc"
UNITS = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}


def _kernels(text):
    """name -> (parameter list, body) of every kernel of a file"""
    found = {}
    for m in re.finditer(r"__global__ .*?(\w+)\(((?:[^()]|\([^()]*\))*)\) \{\n(.*?)\n\}", text, re.S):
        head = text[m.start():m.start(2)]
        name = re.findall(r"(\w+)\($", head)[-1]
        found[name] = (text[m.start(2):m.end(2)], m.group(3))
    return found


KERNELS = {name: (unit, *k) for unit, text in UNITS.items() for name, k in _kernels(text).items()}
CHAINED = sorted(name for name, (_, _, body) in KERNELS.items() if "chain_wait()" in body)


def test_every_kernel_is_found():
    assert sum(len(re.findall(r"__global__", text)) for text in UNITS.values()) == len(KERNELS)
    for must in ("predict_keys_kernel", "build_friends_kernel", "compute_delta_kernel", "cell_gather_kernel",
                 "counting_scan_kernel", "crowded_cells_kernel", "adj_scaling_kernel"):
        assert must in CHAINED


@pytest.mark.parametrize("name", CHAINED)
def test_the_wait_comes_first_and_nothing_passes_it(name):
    unit, parameters, body = KERNELS[name]
    assert body.lstrip().startswith("chain_wait();")
    assert "__restrict__" not in parameters
    assert not re.search(r"__ldg|\.nc\b|__restrict__", body)


@pytest.mark.parametrize("unit", ["pbf_device.cuh", "pbf_kernels.cu", "pbf_adjoint.cu"])
def test_shared_helpers_load_plainly(unit):
    assert not re.search(r"__ldg|\.nc\b|__restrict__", UNITS[unit])


def test_no_other_kernel_is_launched_early():
    """A kernel without the wait is launched by <<<>>>, which waits for the one ahead."""
    early = set()
    for text in UNITS.values():
        for m in re.finditer(r"(?:launch_chained\(|auto k = |cudaLaunchKernelEx\(&cfg, )(.*?);", text, re.S):
            early |= set(re.findall(r"\w+_kernel", m.group(1)))
    assert early and early <= set(CHAINED)
