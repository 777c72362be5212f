"""Window sums of the step partials and the per-particle end of the loads, at the sizes where their
one-cluster forms could go wrong: no rows, fewer rows than groups, remainders of the eight-row blocks,
many rows; one particle, a warp's and a cluster's worth, and both sides of the count above which the
loads take a kernel over all particles."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [0, 1, 8, 31, 32, 33, 255, 256, 257, 2047, 2048, 2368, 20000]


def test_window_sums_of_any_row_count():
    import torch

    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200.engine import stream_handle, struct_to_device, vp

    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(2)
    arr = (nat.PscWindow * len(ROWS))()
    keep, want, scale = [], [], []
    for k, n in enumerate(ROWS):
        tiles = n // nat.PARTIAL_ROWS + 1
        a = np.full((1 + tiles * nat.PARTIAL_ROWS, nat.NRED), np.nan)  # rows past the count are not read
        a[0, 0] = n
        a[1:1 + n] = rng.normal(0, 1, (n, nat.NRED)) * 10.0 ** rng.integers(-6, 6, (n, nat.NRED))
        t = torch.from_numpy(a).to(dev)
        keep.append(t)
        arr[k].partials = t.data_ptr()
        arr[k].tile_count = tiles
        want.append(a[1:1 + n].sum(0))
        scale.append(np.abs(a[1:1 + n]).sum(0))
    out = torch.full((len(ROWS), nat.NRED), np.nan, dtype=torch.float64, device=dev)
    table = struct_to_device(arr, dev)
    for _ in range(2):  # a second reduction of the same partials repeats it
        nat.call("psc_reduce_windows", vp(table), len(ROWS), vp(out), stream_handle(dev))
        got = out.cpu().numpy()
        # a sum of n terms in any order: at most n roundings of half an ulp of the absolute sum
        bound = (np.array(ROWS)[:, None] + 1) * 2.0 ** -53 * np.array(scale)
        assert np.all(np.abs(got - np.array(want)) <= bound)


@pytest.mark.parametrize("P", [0, 1, 33, 256, 257, 4096, 4097])
def test_load_diagnostics_of_any_particle_count(P):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200.handle import BatchHandle, SolverHandle, make_config

    rng = np.random.default_rng(P)
    n = 24
    p = np.zeros((P, 10))
    p[:, 0:3] = rng.uniform(0, n, (P, 3))
    p[:, 3] = rng.uniform(0.6, 1.1, P)
    p[:, 4:7] = rng.normal(0, 1e-3, (P, 3))
    cfg = make_config((n,) * 3, tau=0.8, force=(0.0, 0.0, 1e-6), subsamples=3, store=nat.STORE_F32)
    s = SolverHandle(cfg)
    b = BatchHandle([cfg, cfg], graph_steps=0)
    s.set_particles(p)
    b.set_particles_all([p, p[: P // 2]])
    for _ in range(4):  # the fourth call replays recorded launches and reads a step run ahead
        d = s.step(1, nat.RUN_DIAG).diag
        b.step(1, nat.RUN_DIAG)
    for F, T, d in ((*s.loads(), d), (*b.loads(0), b.diag(0)), (*b.loads(1), b.diag(1))):
        ulp = 2.0 ** -52 * (len(F) + 8)
        assert np.all(np.abs(np.array(d.force_sum) - F.sum(0)) <= ulp * np.abs(F).sum(0) + 1e-300)
        for value, v in ((d.max_force, F), (d.max_torque, T)):
            norm = np.sqrt((v * v).sum(1)).max() if len(v) else 0.0
            assert abs(value - norm) <= 4 * 2.0 ** -52 * norm
    Fs, Ts = s.loads()
    Fb, Tb = b.loads(0)
    assert np.array_equal(Fs, Fb) and np.array_equal(Ts, Tb)
    assert P == 0 or np.abs(Fs).sum() > 0.0
    s.close()
    b.close()


@pytest.mark.parametrize("check_every,max_steps", [(1, 1), (1, 2), (1, 7), (4, 9), (5, 10), (50, 20)])
def test_convergence_rows_are_the_last_steps(check_every, max_steps):
    """A loop that never converges leaves the state, sums, loads and residual of its last step."""
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import windows as wgen
    from particuology_hydraulic_penalty_b200.handle import SolverHandle, make_config

    w = wgen.make_window(20, "skeleton", 3)
    cfg = make_config((20,) * 3, tau=0.72, force=(0.0, 0.0, 1e-6), subsamples=2, store=nat.STORE_F64_EXACT)
    a, b = SolverHandle(cfg), SolverHandle(cfg)
    for h in (a, b):
        h.set_particles(w.particles)
        h.step(1, nat.RUN_DIAG)
    prev = b.diag().mean_uz
    for _ in range(max_steps):
        st = b.step(1, nat.RUN_DIAG)
        prev, before = st.diag.mean_uz, prev
    r = a.converge(max_steps, 0.0, 1, check_every)
    assert r.steps_done == max_steps and not r.converged
    assert r.diag.mean_uz == prev
    want = np.inf if max_steps == 1 else abs(prev - before) / abs(prev)
    assert r.residual == want
    assert np.array_equal(a.field(nat.FIELD_F), b.field(nat.FIELD_F))
    assert np.array_equal(a.field(nat.FIELD_IMB_Z), b.field(nat.FIELD_IMB_Z))
    for x, y in zip(a.loads(), b.loads()):
        assert np.array_equal(x, y)
    assert r.diag.momentum_residual == b.diag().momentum_residual
    assert tuple(r.diag.imb_sum) == tuple(b.diag().imb_sum)
    a.close()
    b.close()
