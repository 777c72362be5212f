"""Results on their way to the host (csrc/solver.cu over stand-ins of the CUDA calls): where no page-locked memory
is to be had, fields and loads arrive through pageable memory, and no error is left for a later call."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("g++ or the CUDA headers not available")
    exe = tmp_path_factory.mktemp("results") / "results_host"
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffunction-sections", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "particuology_hydraulic_penalty_b200" / "csrc"), "-I", str(CUDA),
                    str(ROOT / "tests" / "native" / "results_host.cpp"), "-Wl,--gc-sections",
                    "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe)], check=True)

    def call(*args):
        out = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=60, check=True).stdout
        bad, copied, pinned, waits = map(int, out.split())
        return {"bad": bad, "copied": copied, "pinned": pinned, "waits": waits}

    return call


@pytest.mark.parametrize("no_pinned", [0, 1])
def test_fields_arrive(run, no_pinned):
    assert run("fields", no_pinned)["bad"] == 0


@pytest.mark.parametrize("no_pinned", [0, 1])
@pytest.mark.parametrize("P", [1, 300, 60000])  # 60000: 2.9 MB of loads, more than the page-locked ring
def test_loads_arrive(run, no_pinned, P):
    assert run("loads", no_pinned, 5, P, 0, 1, 2, 4, 3, 1, 0)["bad"] == 0
