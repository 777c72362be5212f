"""Chained launches of the paths that read what the launch ahead wrote: open-x steps (the inlet reads the node's own
populations again) and reverse steps give the bits of launches made one by one."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = 40


@pytest.mark.parametrize("n", [6, 26])
@pytest.mark.parametrize("precision", ["fp64-exact", "fp64", "fp32", "fp16"])
def test_open_x_steps(n, precision):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    dev = torch.device("cuda", 0)
    store = eng.store_mode(precision)
    parts = np.zeros((1, 10))
    parts[0, :4] = [n * 0.5, n * 0.4, n * 0.6, n * 0.25]
    geo = eng.DeviceGeometry((n,) * 3, 2, dev, want_level=store != nat.STORE_F64_EXACT)
    geo.set_particles(parts)
    geo.rebuild()

    def run(wait):
        win = eng.LatticeWindow((n,) * 3, 0.8, (0.0, 0.0, 1e-6), 2, store, None, dev,
                                inlet=(1.0, (0.004, 0.0005, -0.0003)))
        win.bind_geometry(geo)
        for _ in range(STEPS):
            win.step(nat.STEP_IMB)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return win.f[win.cur].cpu().view(torch.uint8).numpy().tobytes(), win.imb.cpu().numpy().tobytes()

    want = run(True)
    assert run(False) == want and run(False) == want


# even nz: two cells per thread; 6^3: fewer CTAs than SMs, the next launch's CTAs wait beside the running one's
@pytest.mark.parametrize("shape", [(6, 6, 6), (5, 6, 7), (30, 31, 32)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_reverse_steps(shape, precision):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    dev, stream = torch.device("cuda", 0), eng.stream_handle(torch.device("cuda", 0))
    dtype = torch.float32 if precision == "fp32" else torch.float64
    N = int(np.prod(shape))
    rng = np.random.default_rng(3)
    state = torch.as_tensor(rng.uniform(-0.01, 0.01, 19 * N), device=dev).to(dtype)
    seed = torch.as_tensor(rng.uniform(-1.0, 1.0, 19 * N), device=dev).to(dtype)
    solid = torch.as_tensor(np.where(rng.random(N) < 0.5, 0.0, rng.random(N)), device=dev)

    def run(wait):
        lam = [seed.clone(), torch.zeros_like(seed)]
        dK = torch.zeros(N, dtype=torch.float64, device=dev)
        args = []
        for k in (0, 1):
            a = nat.PscAdjointArgs()
            a.nx, a.ny, a.nz = shape
            a.store, a.tau, a.kappa = eng.store_mode(precision), 0.8, 1.0
            a.force[0], a.dir[0] = 1e-4, 1.0
            for name, t in (("solid", solid), ("dKdB", dK), ("dKdsolid", dK), ("state", state), ("lam_in", lam[k]),
                            ("lam_out", lam[1 - k])):
                setattr(a, name, eng.vp(t))
            args.append(a)
        for k in range(STEPS):
            nat.call("psc_adjoint_step", ctypes.byref(args[k & 1]), stream)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return lam[STEPS & 1].cpu().numpy().tobytes(), dK.cpu().numpy().tobytes()

    want = run(True)
    assert run(False) == want and run(False) == want
