"""CPU check of the collision that the deviation kernels run (csrc/collide.cuh, collide_v) in FP32: two cells at once
in the packed form are the bits of the cells one by one, and both equal the oracle's collision to FP32 round-off."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import psc_oracle as orc

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "particuology_hydraulic_penalty_b200" / "csrc"


@pytest.fixture(scope="module")
def cells(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("packed") / "collide_packed.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(CSRC),
                    str(ROOT / "tests" / "native" / "collide_packed.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    F = ctypes.POINTER(ctypes.c_float)
    lib.packed_cells.argtypes = [ctypes.c_int] * 2 + [ctypes.c_double] * 5 + [ctypes.c_int] + [F] * 4

    def run(packed, moving, tau, tau_minus, force, g, solid, us):
        n = g.shape[1]
        out = np.zeros((26, n), np.float32)
        lib.packed_cells(packed, moving, tau, tau_minus, *force, n, *(a.ctypes.data_as(F) for a in (g, solid, us, out)))
        return out

    return run


@pytest.mark.parametrize("tau_minus", [0.0, 0.625 + 0.5])
@pytest.mark.parametrize("moving", [0, 1])
def test_packed_cells(cells, moving, tau_minus):
    rng = np.random.default_rng(21)
    n, tau, force = 4096, 0.8, (1e-6, 2e-7, -3e-7)
    g = np.ascontiguousarray(rng.normal(0, 1e-3, (19, n)) * orc.W[:, None], np.float32)
    solid = rng.choice([0.0, 1.0, 0.125, 0.5, 0.984375], size=n).astype(np.float32)
    us = rng.normal(0, 1e-3, (3, n)).astype(np.float32)
    two = cells(1, moving, tau, tau_minus, force, g, solid, us)
    each = cells(0, moving, tau, tau_minus, force, g, solid, us)
    assert np.array_equal(two.view(np.int32), each.view(np.int32))
    shp = (n, 1, 1)
    g64, s64 = g.astype(np.float64).reshape(19, *shp), solid.astype(np.float64).reshape(shp)
    if tau_minus > 0.0:
        if moving:
            return  # (the oracle's TRT extension has no moving solid)
        ref = orc.collide_trt_deviation(g64, s64, tau, tau_minus, force).reshape(19, n)
    else:
        post, imb = orc.collide(g64 + orc.W[:, None, None, None], s64,
                                us.astype(np.float64).reshape(3, *shp) if moving else None, tau, force)
        ref = post.reshape(19, n) - orc.W[:, None]
        # sums of at most forty terms of at most 2 B w (|g| / w + 3 |u| + 3 |us|) <= 0.02
        assert np.abs(each[23:] - imb.reshape(3, n)).max() <= 40 * 2.0 ** -24 * 0.02
    # about thirty roundings of terms of at most w (rho - 1, 3 u, 3 us) / (tau, tau_minus) <= 0.02
    assert np.abs(each[:19] - ref).max() <= 30 * 2.0 ** -24 * 0.02
