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
    assert run("loads", no_pinned, 5, P, 0, 1, 2, 4, 3, 1, 0, "step", 3, 3, 0, 1, 2, 4, 0, "step", 4, 0)["bad"] == 0


@pytest.mark.parametrize("values", [1, 100 ** 3, 160 ** 3])
def test_a_field_asks_for_less_than_a_mapping_of_page_locked_memory(run, values):
    """Page-locking takes longer than a field's transfer, per 2 MB in which smaller allocations share a place."""
    got = run("field", 0, values)
    assert got["bad"] == 0 and got["pinned"] <= 512 << 10


WINDOW = 2 * 3 * 50 * 8  # bytes of one window's loads


def test_reading_two_windows_of_many_brings_a_few(run):
    got = run("loads", 0, 400, 1000, 17, "step", 17, 200)  # 19 MB in all
    assert got["bad"] == 0 and got["copied"] <= 9 * 20 * WINDOW and got["pinned"] <= 512 << 10


def test_the_reads_after_a_batchs_first_step_are_single(run):
    """No page-locked room for all windows before the loads of a second step are read."""
    got = run("loads", 0, 24, 700, *range(24))
    assert got["bad"] == 0 and got["pinned"] <= 14 * WINDOW and got["copied"] == 24 * 14 * WINDOW


@pytest.mark.parametrize("order", [1, -1])
@pytest.mark.parametrize("P", [100, 700, 9000])  # 115 KB, 0.8 and 10 MB of loads
def test_a_batch_asks_for_page_locked_memory_once(run, P, order):
    """A free and a second allocation wait for the device.  Read in turn, up or down, loads beyond the room come over
    once, in pieces of the room (the last of them may reach around)."""
    got = run("loads", 0, 24, P, 0, "step", *range(24)[::order])
    window, room = 48 * P, 512 << 10
    assert got["bad"] == 0 and got["pinned"] <= min(24 * window, room)
    assert got["copied"] <= 24 * window + max(window, min(room, 23 * window))
    assert got["waits"] <= 2 + 24 // min(room // window, 24) + 1


def test_windows_of_more_than_the_room(run):
    got = run("loads", 0, 3, 12000, 0, "step", 0, 1, 2, 0)
    assert got["bad"] == 0 and got["copied"] == 4 * 48 * 12000


@pytest.mark.parametrize("order", ["up", "down", "mixed", "same"])
@pytest.mark.parametrize("nwin", [1, 2, 8, 9, 24, 200])
def test_reading_windows_takes_few_transfers(run, nwin, order):
    """Each transfer brings eight times as many windows as the one before (1, 8, 64, ...) until one brings all,
    in whatever order they are asked for: bytes and waits do not grow with the reads."""
    reads = {"up": list(range(nwin)), "down": list(range(nwin))[::-1], "mixed": [k * 7 % nwin for k in range(nwin)],
             "same": [nwin // 2] * 5}[order]
    got = run("loads", 0, nwin, 50, 0, "step", *reads, *reads)
    transfers = 1 + sum(8 ** k < nwin for k in range(4))
    assert got["bad"] == 0
    assert got["waits"] <= (1 if order == "same" else transfers)
    assert got["copied"] <= (1 if order == "same" else sum(min(8 ** k, nwin) for k in range(transfers))) * WINDOW
