"""Moments of the exact kernels without a collision, under body forces below the range of their branch-free divisions.

Populations that balance pair by pair leave a momentum of F / 2 alone, so u = F / (2 rho) is a quotient
whose numerator may be subnormal or so small that the branch-free form's residual underflows: those
cells take the general division, as they do in a step."""

import numpy as np
import pytest
import torch

from oracle import psc_oracle as orc

pytestmark = pytest.mark.gpu

# the branch-free quotient is off by a bit for about one cell in ten at 1e-308; the others lie beside
FORCES = [(0.0, 0.0, 1.3e-305), (0.0, 0.0, 1.7e-308), (0.0, 1.1e-310, 0.0), (1.9e-308, -1.2e-308, 1.4e-305),
          (0.0, 0.0, 2e-7)]
N = 20


def _balanced(rng):
    """rho between 0.4 and 2 and pairwise equal populations: every momentum sum cancels exactly."""
    a = rng.uniform(0.4, 2.0, (N, N, N))
    f = orc.W[:, None, None, None] * a
    for k in range(9):
        f[2 * k + 2] = f[2 * k + 1]
    return f


@pytest.mark.parametrize("force", FORCES)
def test_moments_pass(force):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    dev = torch.device("cuda", 0)
    f = _balanced(np.random.default_rng(5))
    geo = eng.DeviceGeometry((N,) * 3, 2, dev, want_level=False)
    geo.set_particles(np.zeros((0, 10)))
    geo.rebuild()
    win = eng.LatticeWindow((N,) * 3, 0.72, force, 2, nat.STORE_F64_EXACT, None, dev)
    win.bind_geometry(geo)
    win.load_post_stream_f(torch.as_tensor(f))
    win.moments_pass()
    got = win.moments.cpu().numpy().reshape(4, N, N, N)
    for a, b in zip(got, orc.moments(f, force)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("force", FORCES)
def test_bounceback_moments(force):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    dev = torch.device("cuda", 0)
    f = _balanced(np.random.default_rng(6))
    src = torch.as_tensor(np.ascontiguousarray(orc.unstream_pull(f)), device=dev)
    solid = torch.zeros(N ** 3, dtype=torch.uint8, device=dev)
    mom = torch.empty(4 * N ** 3, dtype=torch.float64, device=dev)
    nat.call("psc_bounceback_step", eng.vp(src), None, eng.vp(solid), N, N, N, 0.8, *force, nat.STEP_MOMENTS,
             eng.vp(mom), eng.stream_handle(dev))
    got = mom.cpu().numpy().reshape(4, N, N, N)
    for a, b in zip(got, orc.moments(f, force)):
        assert np.array_equal(a, b)
