"""Geometries rebuilt for many windows in the same launches equal those of one window at a time."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _particles(rng, count, edge):
    p = np.zeros((count, 10))
    p[:, :3] = rng.random((count, 3)) * edge
    p[:, 3] = 0.6 + 1.5 * rng.random(count)
    p[:, 4:] = rng.normal(size=(count, 6)) * 1e-4
    return p


# 13 and 25: more windows than one launch takes; one window of each has no particles; two values of S
@pytest.mark.parametrize("count", [1, 2, 13, 25])
@pytest.mark.parametrize("precision", ["fp64-exact", "fp32"])
def test_batch_rebuild_equals_single_windows(count, precision):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng
    from particuology_hydraulic_penalty_b200.handle import BatchHandle, SolverHandle, make_config

    rng = np.random.default_rng(count)
    # 8 x 16 x 16 cells are one block of the scan, 12 x 13 x 14 a bit more; 40 x 26 x 30 several
    shapes = [[(8, 16, 16), (12, 13, 14), (40, 26, 30), (6, 7, 9)][k % 4] for k in range(count)]
    cfg = [make_config(sh, tau=0.8, force=(1e-5, 0.0, 0.0), subsamples=2 + (k // 5) % 2, store=eng.store_mode(precision),
                       static_geometry=False, device_index=0) for k, sh in enumerate(shapes)]
    b = BatchHandle(cfg)
    one = [SolverHandle(c) for c in cfg]
    for step in range(3):
        sets = [_particles(rng, 0 if k == 1 else 3 + 7 * ((k + step) % 5), min(sh)) for k, sh in enumerate(shapes)]
        b.set_particles_all(sets)
        b.step(1, nat.RUN_DIAG)
        for k, h in enumerate(one):
            h.set_particles(sets[k])
            h.step(1, nat.RUN_DIAG)
            for which in (nat.FIELD_SOLID, nat.FIELD_ALPHA_SUM, nat.FIELD_US_X, nat.FIELD_US_X + 2, nat.FIELD_UX):
                assert np.array_equal(b.field(k, which), h.field(which)), (step, k, which)
            for got, want in zip(b.loads(k), h.loads()):
                assert np.array_equal(got, want)


def test_scan_of_many_blocks():
    """More blocks than add up their predecessors by themselves: 2049 x 2048 cells and a few."""
    import torch

    from particuology_hydraulic_penalty_b200 import engine as eng

    shape = (163, 161, 160)  # 2050.2 blocks of 2048 cells
    parts = np.zeros((2, 10))
    parts[:, :4] = [[1.5, 1.5, 1.5, 1.2], [161.4, 159.2, 158.3, 1.4]]
    geo = eng.DeviceGeometry(shape, 2, torch.device("cuda", 0), want_level=False)
    geo.set_particles(parts)
    geo.rebuild()
    got = geo.alpha_sum.cpu().numpy().reshape(shape)
    want = np.zeros(shape)
    offs = (np.arange(2) + 0.5) / 2
    for x, y, z, r in parts[:, :4]:
        g = [np.arange(n)[:, None] + offs[None, :] - c for n, c in zip(shape, (x, y, z))]
        lo = [int(max(0, np.floor(c - r - 1))) for c in (x, y, z)]
        hi = [int(min(n, np.ceil(c + r + 1))) for n, c in zip(shape, (x, y, z))]
        s = tuple(slice(a, e) for a, e in zip(lo, hi))
        d2 = (g[0][s[0]][:, :, None, None, None, None] ** 2 + g[1][s[1]][None, None, :, :, None, None] ** 2
              + g[2][s[2]][None, None, None, None, :, :] ** 2)
        want[s] += (d2 <= r * r).sum(axis=(1, 3, 5)) / 8.0
    assert np.array_equal(got, want) and want.max() > 0
