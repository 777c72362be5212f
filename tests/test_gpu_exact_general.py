"""The exact FP64 kernels outside the range of their branch-free arithmetic, and at its edges.

Cells whose populations, force or solid velocity leave that range take the general arithmetic
instead; either way the populations, moments and IMB momentum are the oracle's, bit for bit, on
windows whose last tile is ragged and with forces along an axis and across axes."""

import numpy as np
import pytest

from oracle import psc_oracle as orc
from oracle import voxel_oracle as vo

pytestmark = pytest.mark.gpu

ODD = [0.0, 1e-320, 1e-300, 2.0 ** -15, np.nextafter(2.0 ** -15, 0.0), np.nextafter(2.0, 0.0), 2.0, 40.0, -1 / 36,
       1e150]


def _particles(n, moving, rng):
    p = np.zeros((5, 10))
    p[:, 0:3] = rng.uniform(0, n, (5, 3))
    p[:, 3] = rng.uniform(1.2, 2.6, 5)
    if moving:
        p[:3, 4:7] = rng.normal(0, 1e-3, (3, 3))
        p[2, 7:10] = rng.normal(0, 1e-4, 3)
        p[1, 4] = 1e-250  # outside the range the branch-free forms take
    return p


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("n,force", [(8, (0.0, 0.0, 2e-7)), (9, (0.0, 3e-6, 0.0)), (17, (1e-6, 0.0, 0.0)),
                                     (9, (3e-7, -2e-7, 5e-7)), (9, (0.0, 0.0, 1e-310)), (9, (0.0, 0.0, 0.0))])
def test_exact_step_with_odd_populations(n, force, moving):
    from particuology_hydraulic_penalty_b200 import SparsePscD3Q19

    rng = np.random.default_rng(n)
    parts = _particles(n, moving, rng)
    f = orc.W[:, None, None, None] * (1.0 + rng.normal(0, 1e-2, (19, n, n, n)))
    where = rng.random(f.shape) < 0.004  # about one cell in thirteen
    f[where] = rng.choice(ODD, int(where.sum()))
    kw = dict(tau=0.72, subsamples=3, force=force, static_geometry=True)
    o = orc.OracleSolver(n, parts, **kw)
    g = SparsePscD3Q19(n, parts, **kw)
    o.f = f.copy()
    g.f = f
    with np.errstate(all="ignore"):
        o.collide_stream_psc()
    g.collide_stream_psc()
    assert np.array_equal(g.f, o.f, equal_nan=True)
    for a, b in ((g.rho, o.rho), (g.ux, o.ux), (g.uy, o.uy), (g.uz, o.uz), (g.imb_mx, o.imb[0]), (g.imb_my, o.imb[1]),
                 (g.imb_mz, o.imb[2])):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("n,force_z", [(7, 1e-6), (12, 1e-310), (13, 2e-4)])
def test_voxel_solver_equals_the_oracle(n, force_z):
    from particuology_hydraulic_penalty_b200 import voxel_lbm

    solid = np.random.default_rng(n).random((n, n, n)) < 0.3
    a = voxel_lbm.run_lbm(solid, 0.8, force_z, 9, return_fields=True)
    b = vo.run_lbm(solid, 0.8, force_z, 9, return_fields=True)
    for k in ("ux", "uy", "uz"):
        assert np.array_equal(a[k], b[k]), k
