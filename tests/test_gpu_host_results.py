"""Fields and loads on the host: pieces of the page-locked ring, and a batch's windows in any order."""

import numpy as np
import pytest

from oracle.psc_oracle import C, W

pytestmark = pytest.mark.gpu


def _solver(n, precision, parts):
    from particuology_hydraulic_penalty_b200.psc3d import SparsePscD3Q19

    return SparsePscD3Q19(n, parts, subsamples=2, body_force_z=1e-6, static_geometry=True, precision=precision)


# 65536 floats or 32768 doubles to a piece: one, one and a bit, more than the ring's eight
@pytest.mark.parametrize("n", [3, 32, 40, 41, 84])
@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp16"])
def test_fields_in_pieces(n, precision):
    """Every cell's density and velocity against the moments of the populations the solver returns."""
    parts = np.zeros((1, 10))
    parts[0, :4] = n / 2, n / 2, n / 2, n / 4
    s = _solver(n, precision, parts)
    for _ in range(3):
        diag = s.collide_stream_psc()
    f, uz, rho = s.f, s.uz, s.rho
    assert uz.shape == (n, n, n) and uz.dtype == np.float64
    # 19 terms in the window's arithmetic; the momentum is a sum of 10 deviations below 1e-4
    eps = 2.0 ** -52 if precision == "fp64" else 2.0 ** -23
    assert np.abs(rho - f.sum(axis=0)).max() <= 19 * eps
    want = np.einsum("i,i...->...", C[:, 2].astype(float), f - W[:, None, None, None]) / rho + 0.5e-6 / rho
    assert np.abs(uz - want).max() <= 100 * eps * 1e-4 + 1e-15
    assert abs(uz.mean() - diag["mean_uz"]) <= 1e-5 * abs(diag["mean_uz"])


@pytest.mark.parametrize("order", [[0, 1, 2, 3], [3, 3, 0, 1, 2], [2], [1, 0, 1, 3, 2]])
def test_batch_loads_any_order(order):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng
    from particuology_hydraulic_penalty_b200.handle import BatchHandle, make_config

    rng = np.random.default_rng(3)
    shapes, sets = [(12, 12, 12), (9, 10, 14), (16, 16, 16), (8, 8, 8)], []
    for k, sh in enumerate(shapes):
        p = np.zeros(((5, 1, 40, 0)[k], 10))
        p[:, :3] = rng.random((len(p), 3)) * min(sh)
        p[:, 3] = 1.0 + rng.random(len(p))
        sets.append(p)
    cfg = [make_config(sh, tau=0.8, force=(0.0, 0.0, 1e-5), subsamples=3, store=eng.store_mode("fp32"),
                       static_geometry=True, device_index=0) for sh in shapes]
    b = BatchHandle(cfg)
    b.set_particles_all(sets)
    one = []
    for k in range(4):
        h = BatchHandle(cfg[k:k + 1])
        h.set_particles_all(sets[k:k + 1])
        one.append(h)
    for steps in (2, 1, 1):  # the loads of an earlier step are not returned again
        b.step(steps, nat.RUN_DIAG)
        for h in one:
            h.step(steps, nat.RUN_DIAG)
        for k in order:
            for got, want in zip(b.loads(k), one[k].loads(0)):
                assert got.shape == (len(sets[k]), 3)
                assert np.array_equal(got, want)
        assert np.abs(b.loads(2)[0]).max() > 0.0
