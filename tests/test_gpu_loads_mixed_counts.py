"""A window's loads are the same bits alone and in a batch, whatever the particle counts of the other windows:
particles of many load chunks beside a window above the count at which the loads take a kernel over all particles."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _small(n, count, rng):
    p = np.zeros((count, 10))
    p[:, 0:3] = rng.uniform(0, n, (count, 3))
    p[:, 3] = rng.uniform(0.6, 1.1, count)
    return p


@pytest.mark.parametrize("others", [(4097,), (4096,), (5000, 0, 40)])
@pytest.mark.parametrize("store", ["fp32", "fp64-exact"])
def test_loads_do_not_depend_on_the_other_windows(others, store):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200.engine import store_mode
    from particuology_hydraulic_penalty_b200.handle import BatchHandle, SolverHandle, make_config

    rng = np.random.default_rng(8)
    n = 64
    p = _small(n, 300, rng)
    p[:6, 0:3] = rng.uniform(20, 44, (6, 3))
    p[:6, 3] = [20.0, 17.0, 14.0, 12.0, 9.0, 8.0]  # boxes of 21, 13, 8, 5, 3 and 2 chunks of 4096 cells
    big = make_config((n,) * 3, tau=0.8, force=(1e-6, 2e-6, -1e-6), subsamples=3, store=store_mode(store))
    lil = make_config((24,) * 3, tau=0.8, force=(1e-6, 0.0, 0.0), subsamples=3, store=store_mode(store))
    alone = SolverHandle(big)
    batch = BatchHandle([big] + [lil] * len(others), graph_steps=0)
    alone.set_particles(p)
    batch.set_particles_all([p] + [_small(24, k, rng) for k in others])
    for _ in range(3):
        d = alone.step(1, nat.RUN_DIAG).diag
        batch.step(1, nat.RUN_DIAG)
    for x, y in zip(alone.loads(), batch.loads(0)):
        assert np.abs(x).sum() > 0.0
        assert np.array_equal(x, y)
    # (the window sums behind momentum_residual are added per CTA, whose share of a window depends on the batch)
    assert d.max_force == batch.diag(0).max_force and d.max_torque == batch.diag(0).max_torque
    alone.close()
    batch.close()
