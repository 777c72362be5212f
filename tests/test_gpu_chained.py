"""Steps launched before the step ahead of them has ended give the bits of steps launched one by one."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = 60


def _run(precision, n, kernel, flags, chained):
    """Populations and sums after STEPS steps back to back from a perturbed state, enqueued without a wait."""
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    dev = torch.device("cuda", 0)
    store = eng.store_mode(precision)
    parts = np.zeros((2, 10))
    parts[:, :4] = [[n * 0.3, n * 0.4, n * 0.5, n * 0.2], [n * 0.7, n * 0.6, n * 0.2, n * 0.15]]
    geo = eng.DeviceGeometry((n,) * 3, 3, dev, want_level=store != nat.STORE_F64_EXACT)
    geo.set_particles(parts)
    geo.rebuild()
    win = eng.LatticeWindow((n,) * 3, 0.8, (1e-5, 2e-6, 0.0), 3, store, None, dev)
    win.bind_geometry(geo)
    win.ensure_fields(True, False)
    plan = "psc_plan_pair_tiles" if kernel == nat.KERNEL_PAIR else "psc_plan_tiles"
    tables, rows = [], []
    for src in (0, 1):
        d = win.struct(src)
        total = ctypes.c_int64(0)
        args = (ctypes.byref(d), 1) + (() if kernel == nat.KERNEL_PAIR else (0,)) + (ctypes.byref(total),)
        nat.call(plan, *args)
        part = torch.zeros((1 + total.value * nat.PARTIAL_ROWS) * nat.NRED, dtype=torch.float64, device=dev)
        d.partials = part.data_ptr()
        rows.append(part)
        tables.append((eng.struct_to_device((nat.PscWindow * 1)(d), dev), total.value))
    cfg = nat.PscLaunch(0, 1, kernel, 0, 0)
    sums = torch.zeros((STEPS, nat.NRED), dtype=torch.float64, device=dev)
    stream = eng.stream_handle(dev)
    for k in range(STEPS):
        t, total = tables[k & 1]
        fl = nat.STEP_COLLIDE | flags | (nat.STEP_CHAINED if chained else 0)
        nat.call("psc_step_windows_ex", store, eng.vp(t), 1, total, fl, ctypes.byref(cfg), stream)
        if flags & nat.STEP_REDUCE:
            nat.call("psc_reduce_windows", eng.vp(t), 1, eng.vp(sums[k]), stream)
        if not chained:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    return win.f[STEPS & 1].cpu().view(torch.uint8).numpy().tobytes(), sums.cpu().numpy().tobytes()


# 6: fewer tiles than SMs, the next steps wait beside the running one; 40: more than one tile per CTA
@pytest.mark.parametrize("n", [6, 24, 40])
@pytest.mark.parametrize("precision,kernel", [("fp64-exact", 0), ("fp64", 1), ("fp32", 1), ("fp32", 3), ("fp16", 3)])
@pytest.mark.parametrize("reduce", [False, True])
def test_chained_steps(n, precision, kernel, reduce):
    from particuology_hydraulic_penalty_b200 import _native as nat

    flags = (nat.STEP_IMB | nat.STEP_REDUCE) if reduce else 0
    want = _run(precision, n, kernel, flags, False)
    for _ in range(3):
        assert _run(precision, n, kernel, flags, True) == want


@pytest.mark.parametrize("shape", [(5, 6, 7), (24, 24, 24), (31, 64, 40)])
@pytest.mark.parametrize("steps", [0, 1, 2, 41])
def test_bounceback_steps(shape, steps):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng

    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(5)
    N = int(np.prod(shape))
    solid = torch.as_tensor((rng.random(N) < 0.2).astype(np.uint8), device=dev)
    stream = eng.stream_handle(dev)

    def run(chained):
        f = [torch.zeros(19 * N, dtype=torch.float64, device=dev) for _ in range(2)]
        mom = torch.zeros(4 * N, dtype=torch.float64, device=dev)
        nat.call("psc_init_equilibrium", nat.STORE_F64_EXACT, 1.0, eng.vp(f[0]), N, stream)
        if chained:
            nat.call("psc_bounceback_steps", eng.vp(f[0]), eng.vp(f[1]), eng.vp(solid), *shape, 0.8, 1e-5, 0.0, 2e-5,
                     steps, eng.vp(mom), stream)
        else:
            for k in range(steps + 1):
                last = k == steps
                nat.call("psc_bounceback_step", eng.vp(f[k & 1]), None if last else eng.vp(f[1 - (k & 1)]),
                         eng.vp(solid), *shape, 0.8, 1e-5, 0.0, 2e-5, nat.STEP_MOMENTS if last else nat.STEP_COLLIDE,
                         eng.vp(mom) if last else None, stream)
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return f[steps & 1].cpu().numpy().tobytes(), mom.cpu().numpy().tobytes()

    assert run(True) == run(False)
