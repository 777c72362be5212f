"""Loads and diagnostics asked for between new particles and the step that voxelises them, in a window that has
held no particle so far: refused, not answered with zeros.  Particles that all lie outside the window have a
geometry without entries; their loads are zero."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _particles(centre):
    p = np.zeros((3, 10))
    p[:, 0:3] = centre
    p[:, 0] += [0.0, 3.0, 6.0]
    p[:, 3] = 1.4
    return p


@pytest.mark.parametrize("store", ["fp64-exact", "fp32"])
def test_new_particles_before_the_first_geometry(store):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200.engine import store_mode
    from particuology_hydraulic_penalty_b200.handle import SolverHandle, make_config

    h = SolverHandle(make_config((16,) * 3, tau=0.8, force=(0.0, 0.0, 1e-5), subsamples=2, store=store_mode(store),
                                 static_geometry=False))
    h.set_particles(np.zeros((0, 10)))
    for _ in range(3):
        h.step(1, nat.RUN_DIAG)
    h.set_particles(_particles([4.0, 8.0, 8.0]))
    for call in (h.loads, h.diag):
        with pytest.raises(nat.PscError, match="null array"):
            call()
    for _ in range(3):
        h.step(1, nat.RUN_DIAG)
    assert np.abs(h.loads()[0]).sum() > 0.0
    h.close()


def test_particles_outside_the_window():
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200.handle import SolverHandle, make_config

    h = SolverHandle(make_config((16,) * 3, tau=0.8, force=(0.0, 0.0, 1e-5), subsamples=2, store=nat.STORE_F64_EXACT,
                                 static_geometry=False))
    h.set_particles(_particles([40.0, 40.0, 40.0]))
    for _ in range(3):
        d = h.step(1, nat.RUN_DIAG).diag
    F, T = h.loads()
    assert F.shape == (3, 3) and not F.any() and not T.any()
    assert d.max_force == 0.0 and d.max_torque == 0.0
    h.close()
