"""run_lbm hands its steps to the library in pieces: a long run can be interrupted between them, and the result
does not depend on where they end."""

import contextlib

import numpy as np
import pytest
import torch

PIECE = 64


@pytest.fixture
def on_the_host(monkeypatch):
    """run_lbm with the device replaced by the host and the library by a recorder of its calls."""
    from particuology_hydraulic_penalty_b200 import voxel_lbm

    calls = []
    monkeypatch.setattr(voxel_lbm, "require_cuda", lambda device: torch.device("cpu"))
    monkeypatch.setattr(voxel_lbm, "stream_handle", lambda device: None)
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())

    def call(name, *args):
        if name == "psc_bounceback_steps":
            steps, moments = int(args[-3]), args[-2]
            calls.append((args[0].value, steps, moments is not None))
            if len(calls) == call.interrupt_at:
                raise KeyboardInterrupt

    call.interrupt_at = 0
    monkeypatch.setattr(voxel_lbm.nat, "call", call)
    return voxel_lbm, calls, call


@pytest.mark.parametrize("steps", [-1, 0, 1, PIECE - 1, PIECE, PIECE + 1, 1000])
def test_pieces(on_the_host, steps):
    voxel_lbm, calls, _ = on_the_host
    voxel_lbm.run_lbm(np.zeros((3, 4, 5), bool), 0.8, 1e-6, steps)
    assert sum(k for _, k, _ in calls) == max(steps, 0)
    assert all(k <= PIECE for _, k, _ in calls)
    assert all(k % 2 == 0 for _, k, _ in calls[:-1])  # the state is back in the first buffer
    assert len({f for f, _, _ in calls}) == 1
    assert [m for _, _, m in calls] == [False] * (len(calls) - 1) + [True]  # the moments come with the last piece


def test_an_interrupt_ends_a_long_run(on_the_host):
    voxel_lbm, calls, call = on_the_host
    call.interrupt_at = 3
    with pytest.raises(KeyboardInterrupt):
        voxel_lbm.run_lbm(np.zeros((3, 4, 5), bool), 0.8, 1e-6, 10 ** 9)
    assert len(calls) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [0, 1, PIECE, PIECE + 1, 3 * PIECE - 1])
def test_pieces_give_the_state_of_one_call(steps):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200 import engine as eng
    from particuology_hydraulic_penalty_b200 import voxel_lbm

    shape, dev = (9, 14, 11), torch.device("cuda", 0)
    N = int(np.prod(shape))
    solid = np.random.default_rng(2).random(shape) < 0.2
    got = voxel_lbm.run_lbm(solid, 0.8, 2e-5, steps, return_fields=True)
    s = torch.as_tensor(solid.astype(np.uint8).reshape(-1), device=dev)
    f = [torch.zeros(19 * N, dtype=torch.float64, device=dev) for _ in range(2)]
    mom = torch.zeros(4 * N, dtype=torch.float64, device=dev)
    st = eng.stream_handle(dev)
    nat.call("psc_init_equilibrium", nat.STORE_F64_EXACT, 1.0, eng.vp(f[0]), N, st)
    nat.call("psc_bounceback_steps", eng.vp(f[0]), eng.vp(f[1]), eng.vp(s), *shape, 0.8, 0.0, 0.0, 2e-5, steps,
             eng.vp(mom), st)
    want = mom.view(4, *shape).cpu().numpy()
    for k, name in enumerate(("ux", "uy", "uz")):
        assert np.array_equal(got[name], want[1 + k])
