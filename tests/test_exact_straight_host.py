"""CPU check of the branch-free forms of the exact FP64 arithmetic (csrc/d3q19.cuh, csrc/collide.cuh).

The divisions must round as the host's IEEE binary64 division does: on every significand that could
lie within the forms' error of a midpoint (enumerated with exact integers), on random operands over
the range the forms state, and on its edges.  Whole cells must equal the general forms value for value
wherever the range flag is clear, and the flag must be set for operands outside the range."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "particuology_hydraulic_penalty_b200" / "csrc"
TAUS = [0.5000001, 0.51, 0.6, 0.72, 0.75, 0.8, 1.0, 1.2345678901234567, 1.7, 2.0 ** -8, 255.9]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("straight") / "exact_straight.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(CSRC),
                    str(ROOT / "tests" / "native" / "exact_straight.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    D = ctypes.POINTER(ctypes.c_double)
    lib.straight_list.restype = lib.straight_random.restype = ctypes.c_longlong
    lib.straight_list.argtypes = [ctypes.c_int, ctypes.c_double, D, ctypes.c_longlong]
    lib.straight_random.argtypes = [ctypes.c_int, ctypes.c_double, ctypes.c_longlong, ctypes.c_uint64, ctypes.c_int,
                                    ctypes.c_int]
    lib.range_test.argtypes = [ctypes.c_double]
    lib.straight_cells.argtypes = [D, D, D, ctypes.c_int] + [ctypes.c_double] * 4 + [ctypes.c_int] + [D] * 3 + \
        [ctypes.POINTER(ctypes.c_int)] + [D] * 3
    return lib


def _p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _near_midpoints(y):
    """Every x in [1, 2) whose quotient by y lies within 2^-48 ulp of a midpoint of two doubles.

    X, Y the 53-bit integers of x and y, M the odd 54-bit integer of the midpoint: X 2^s = M Y + j with
    s = 53 (X >= Y) or 54, and |j| < Y 2^-48 2^-1 <= 16, so M is -j / Y modulo 2^s (up to Y's factors of 2).
    """
    m, e = np.frexp(y)
    Y = int(m * 2.0 ** 53)
    t = (Y & -Y).bit_length() - 1
    found = []
    for s in (53, 54):
        mod = 1 << (s - min(t, s))
        inv = pow(Y >> t, -1, mod) if mod > 1 else 0
        for j in range(-40, 41):
            if j % (1 << t):
                continue
            M = (-(j >> t) * inv) % mod if mod > 1 else 0
            while M < 1 << 54:
                if M >= 1 << 53 and M & 1:
                    X, rem = divmod(M * Y + j, 1 << s)
                    if rem == 0 and 1 << 52 <= X < 1 << 53 and (X >= Y) == (s == 53):
                        found.append(X * 2.0 ** -52)
                M += mod
                if t > 12:
                    break
    return found


def test_divisors_are_one_third_and_one_ninth_less_one_rounding():
    from fractions import Fraction

    one = 1 - Fraction(1, 2 ** 54)
    assert Fraction(1.0 / 3.0) == one / 3
    assert Fraction((1.0 / 3.0) * (1.0 / 3.0)) == one / 9


@pytest.mark.parametrize("k,y", [(0, 1.0 / 3.0), (1, (1.0 / 3.0) ** 2), (2, 1.0 / 3.0), (3, (1.0 / 3.0) ** 2)] +
                         [(4, t) for t in TAUS] + [(5, t) for t in TAUS])
def test_divisions_round_as_ieee(lib, k, y):
    near = _near_midpoints(y)
    xs = np.array([s * x * 2.0 ** e for x in near for s in (1, -1) for e in (-890, -60, -1, 0, 1, 890)], dtype=float)
    if len(xs):
        assert lib.straight_list(k, y, _p(xs), len(xs)) == 0
    top = 900 if k >= 4 else 960
    edge = np.array([1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.5, 4.0 / 3.0, 2.0 ** -top, 2.0 ** (top - 1), 0.0,
                     5.0 / 3.0, 16.0 / 9.0, 8.0 / 7.0], dtype=float)
    edge = np.concatenate([edge, -edge[edge != 0.0], edge * 2.0 ** -40])
    edge = edge[(np.abs(edge) >= 2.0 ** -top) | (edge == 0.0)]
    assert lib.straight_list(k, y, _p(edge), len(edge)) == 0
    for seed, (lo, hi) in enumerate([(-top, top - 1), (-40, 4), (-2, 1)]):
        assert lib.straight_random(k, y, 300000, 77 + seed, lo, hi) == 0


def test_random_divisors_near_midpoints(lib):
    rng = np.random.default_rng(11)
    for y in np.concatenate([rng.uniform(0.5, 2.0, 200), rng.uniform(0.97, 1.03, 200)]):
        xs = np.array([x * 2.0 ** e for x in _near_midpoints(float(y)) for e in (-30, 0)], dtype=float)
        if len(xs):
            assert lib.straight_list(4, float(y), _p(xs), len(xs)) == 0
            assert lib.straight_list(5, float(y), _p(xs), len(xs)) == 0


def test_range_flag(lib):
    inside = [0.0, -0.0, 1.0, -1.0, 2.0 ** -200, -2.0 ** -200, np.nextafter(2.0 ** 200, 0.0)]
    outside = [np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1030, np.nextafter(2.0 ** -200, 0.0), 2.0 ** 200, 1e308]
    assert [lib.range_test(x) for x in inside] == [0] * len(inside)
    assert [lib.range_test(x) for x in outside] == [1] * len(outside)


def _cells(lib, f, solid, us, moving, tau, force):
    n = f.shape[1]
    a = [np.zeros((19, n)), np.zeros((3, n)), np.zeros((4, n))]
    b = [np.zeros((19, n)), np.zeros((3, n)), np.zeros((4, n))]
    out = np.zeros(n, dtype=np.int32)
    lib.straight_cells(_p(np.ascontiguousarray(f)), _p(np.ascontiguousarray(solid)), _p(np.ascontiguousarray(us)),
                       int(moving), tau, *force, n, *(_p(x) for x in a), out.ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
                       *(_p(x) for x in b))
    return a, b, out


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("force", [(0.0, 0.0, 2e-7), (1e-6, 0.0, 0.0), (3e-7, -2e-7, 5e-7), (0.0, 0.0, 0.0)])
def test_cells_equal_the_general_forms(lib, moving, force):
    rng = np.random.default_rng(3)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)[:, None]
    n = 4000
    f = np.concatenate([w * (1.0 + rng.normal(0, amp, (19, n))) for amp in (0.0, 1e-9, 1e-3)] +
                       [w * rng.uniform(0.01, 3.0, (19, n))], axis=1)
    n = f.shape[1]
    solid = rng.choice([0.0, 1.0, -0.5, 1.5, 0.125, 0.984375, 0.37], size=n)
    us = rng.normal(0, 1e-3, (3, n)) * rng.integers(0, 2, (3, n))
    for tau in (0.51, 0.72, 1.0):
        a, b, out = _cells(lib, f, solid, us, moving, tau, force)
        assert not out.any()
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


def test_cells_outside_the_range_are_flagged_or_equal(lib):
    """Populations, forces and velocities of any size: a cell is flagged or equal (NaN counts as itself)."""
    rng = np.random.default_rng(5)
    n = 6000
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)[:, None]
    f = np.repeat(w, n, axis=1) * (1.0 + rng.normal(0, 1e-2, (19, n)))
    for c in range(n):
        for _ in range(rng.integers(1, 6)):
            f[rng.integers(19), c] = rng.choice([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-300, -1e-310, 1e300, 1e150,
                                                 2.0 ** -901, 1e-200, -1 / 36, 1e-20, 256.0, 300.0, 2.0 ** -15, 2.0,
                                                 np.nextafter(2.0 ** -15, 0.0), np.nextafter(2.0, 0.0)])
    f[:, :19] = 0.0
    f[:, 19:40] = np.nextafter(2.0, 0.0)  # rho about 38
    f[:, 40:60] = 2.0 ** -15  # rho below 2^-8
    solid = rng.choice([0.0, 1.0, 0.5], size=n)
    us = rng.choice([0.0, 1e-3, 1e-320, 1e200, np.inf, 1e-70], size=(3, n))
    with np.errstate(all="ignore"):
        for moving in (False, True):
            for tau, force in ((0.72, (0.0, 0.0, 2e-7)), (0.8, (1e-310, 0.0, 0.0)), (0.8, (0.0, 1e250, 0.0)),
                               (300.0, (0.0, 0.0, 1e-6)), (0.6, (1e-55, -1e-60, 0.0))):
                a, b, out = _cells(lib, f, solid, us, moving, tau, force)
                ok = out == 0
                for x, y in zip(a, b):
                    assert np.array_equal(x[:, ok], y[:, ok], equal_nan=True)
