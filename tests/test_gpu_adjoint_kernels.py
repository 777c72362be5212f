"""The reverse step's kernels (one cell and two cells per thread) and the smooth fraction's, against the FP64
adjoint in numpy, at the sizes and alignments where they change."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import psc_adjoint as adj

pytestmark = pytest.mark.gpu

TAU, F = 0.8, (1e-4, -2e-5, 3e-5)


def _at(a, dtype, shift):
    """Device copy of a, `shift` elements past an allocation's start."""
    buf = torch.zeros(a.size + shift, dtype=dtype, device="cuda")
    buf[shift:] = torch.as_tensor(np.ascontiguousarray(a).ravel(), device="cuda").to(dtype)
    return buf[shift:]


# nz even with every pointer aligned: two cells per thread; 2 is the smallest, 512 cells one block's pairs
@pytest.mark.parametrize("shape,shift", [((1, 1, 2), 0), ((3, 2, 2), 0), ((5, 3, 4), 0), ((4, 8, 16), 0),
                                         ((2, 9, 30), 0), ((2, 9, 30), 1), ((3, 3, 7), 0), ((1, 1, 1), 0),
                                         ((40, 41, 74), 0)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_reverse_step(shape, shift, precision):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    dtype, eps = (torch.float32, 2.0 ** -24) if precision == "fp32" else (torch.float64, 2.0 ** -53)
    rng = np.random.default_rng(7)
    round_ = (lambda x: x.astype(np.float32).astype(np.float64)) if precision == "fp32" else (lambda x: x)
    state = round_(rng.uniform(-0.01, 0.01, (19,) + shape))
    lam = round_(rng.uniform(-1.0, 1.0, (19,) + shape))
    solid = np.where(rng.random(shape) < 0.5, rng.integers(0, 2, shape).astype(float), rng.random(shape))
    before = rng.uniform(-1.0, 1.0, shape)
    S, L = _at(state, dtype, shift), _at(lam, dtype, shift)
    out = torch.full((L.numel() + shift,), float("nan"), dtype=dtype, device="cuda")[shift:]
    al, dB = _at(solid, torch.float64, shift), _at(before, torch.float64, shift)
    a = nat.PscAdjointArgs()
    a.nx, a.ny, a.nz = shape
    a.store, a.tau, a.kappa = eng.store_mode(precision), TAU, 1.0
    for k in range(3):
        a.force[k], a.dir[k] = F[k], float(k == 0)
    ds = torch.zeros_like(dB)
    for name, t in (("solid", al), ("dKdB", dB), ("dKdsolid", ds), ("state", S), ("lam_in", L), ("lam_out", out)):
        setattr(a, name, eng.vp(t))
    nat.call("psc_adjoint_step", ctypes.byref(a), eng.stream_handle(torch.device("cuda", 0)))
    mu, dK = adj.collide_dev_vjp(adj.pull(state), adj.bweight(solid, TAU), lam, TAU, F)
    # each value is a sum of at most ~100 products of order max |lambda| sum(w) (1 + 1/tau); dC/dB has 19 more
    tol = 200.0 * eps * (1.0 + 1.0 / TAU)
    got = out.double().cpu().numpy().reshape(mu.shape)
    assert np.abs(got - adj.pull_T(mu)).max() <= tol
    assert np.abs(dB.cpu().numpy().reshape(shape) - before - dK).max() <= tol


@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 6, 7])
def test_smooth_fraction_and_gradient(S):
    """A particle of several chunks, small ones, one through the corner and one that owns no cell."""
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    n, eps = 24, 0.05
    dev = torch.device("cuda", 0)
    parts = np.zeros((5, 10))
    parts[:, 0:4] = [[11.2, 12.6, 11.9, 9.3], [3.4, 20.1, 5.5, 1.3], [0.2, 0.1, 23.7, 2.5], [60.0, 60.0, 60.0, 1.0],
                     [18.5, 18.5, 18.5, 0.4]]
    geo = eng.DeviceGeometry((n,) * 3, S, dev, want_level=False, smooth_eps=eps)
    geo.set_particles(parts)
    geo.rebuild()
    ent = adj.smooth_alpha(parts, n, S, eps, with_grad=True)
    asum = adj.smooth_solid(parts, n, S, eps)[0]
    # a sample's argument (r - d) / eps carries ~ 4 ulp of d / eps <= 20 / 0.05, and sigma' <= 1/4
    tol = 4.0 * 2.0 ** -52 * (20.0 / eps) * 0.25 * len(parts) + S ** 3 * 2.0 ** -53
    got = geo.alpha_sum.cpu().numpy().ravel()
    assert np.abs(got - asum).max() <= tol

    rng = np.random.default_rng(S)
    gB, gs = rng.uniform(-1, 1, n ** 3), rng.uniform(-1, 1, n ** 3)
    dB, ds = (torch.as_tensor(x, device=dev) for x in (gB, gs))
    a = nat.PscAdjointArgs()
    a.nx = a.ny = a.nz = n
    a.store, a.tau, a.kappa = eng.store_mode("fp64"), TAU, 1.0
    a.solid, a.dKdB, a.dKdsolid = eng.vp(geo.solid), eng.vp(dB), eng.vp(ds)
    part = torch.zeros(geo.cap_chunks * 4, dtype=torch.float64, device=dev)
    grad = torch.full((len(parts), 4), float("nan"), dtype=torch.float64, device=dev)
    g = geo.struct()
    nat.call("psc_adjoint_geometry_grad", ctypes.byref(g), ctypes.byref(a), eng.vp(part), eng.vp(grad),
             eng.stream_handle(dev))
    grad = grad.cpu().numpy()
    cell = np.where((got > 0.0) & (got < 1.0), gB * adj.dbweight(got, TAU) + gs, 0.0)
    for p in range(len(parts)):
        terms = ent[p][2] * cell[ent[p][0]]
        # sigma' turns by less than its argument's error; sigma (1 - sigma) of the oracle loses 2^-53 per sample
        bound = 16.0 * 2.0 ** -52 * (20.0 / eps) * np.abs(terms).sum() + terms.size * 2.0 ** -50 / eps
        assert np.abs(grad[p] - terms.sum(axis=1)).max() <= bound
