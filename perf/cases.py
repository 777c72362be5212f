"""The work that users of this package have it do, as cases that can be timed and checked.

Every case goes through a public entry point: the drop-in solver
(``SparsePscD3Q19``) the way the permeability probe and the DEM-coupled driver
call it, batches of uneven windows (``PscBatch``, ``BatchHandle``), the
differentiable permeability, and the voxel bounce-back solver.  Sizes, relaxation
times, forces and geometries are those of the repository's benchmark, probe,
validation campaign and tests.

Solvers that compute in 32 bits hand their results on as 32-bit numbers here;
the FP64 ones as 64-bit numbers.
"""

from __future__ import annotations

import itertools
import math

import numpy as np
import torch
import torch.utils.checkpoint

from particuology_hydraulic_penalty_b200 import Particle3D, SparsePscD3Q19
from particuology_hydraulic_penalty_b200 import _native as nat
from particuology_hydraulic_penalty_b200 import coupling, voxel_lbm
from particuology_hydraulic_penalty_b200.adjoint import PermeabilityProblem, permeability
from particuology_hydraulic_penalty_b200.batch import PscBatch, WindowSpec
from particuology_hydraulic_penalty_b200.engine import store_mode
from particuology_hydraulic_penalty_b200.handle import BatchHandle, make_config
from particuology_hydraulic_penalty_b200.windows import fcc_skeleton, preload, rsa_fines

KINDS = ("skeleton", "passive", "preloaded")
BATCH_EDGES = (48, 64, 96, 128, 160)
# (the closure residual of the momenta is rounding alone: nothing to compare)
DIAG = ("solid_volume_lu", "mean_uz", "max_force", "max_torque")
BATCH_DIAG = ("solid_volume_lu", "max_force", "max_torque", "permeability", "fluid_volume_lu")


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the probe on a coarse window: latency of one reporting call after the other
        {"name": "probe_exact_24", "path": "probe", "precision": "fp64-exact", "n": 24, "kind": "skeleton",
         "subsamples": 2, "steps": 30},
        # the probe at the usual resolution of a resolution study, in the default (reference) arithmetic
        {"name": "probe_exact_96", "path": "probe", "precision": "fp64-exact", "n": 96, "kind": "preloaded",
         "subsamples": 4, "steps": 60},
        # the probe in single precision on an odd edge
        {"name": "probe_fp32_75", "path": "probe", "precision": "fp32", "n": 75, "kind": "passive",
         "subsamples": 3, "steps": 60},
        # a macro step of the DEM-coupled driver: moved particles, geometry rebuilt, a few steps, loads
        {"name": "coupled_exact_64", "path": "coupled", "precision": "fp64-exact", "n": 64, "kind": "preloaded",
         "subsamples": 3, "steps": 10},
        # the quasi-steady macro step of the same driver: its convergence loop, every step checked
        {"name": "converge_exact_48", "path": "converge", "precision": "fp64-exact", "n": 48, "kind": "preloaded",
         "subsamples": 3, "steps": 40, "check_every": 1},
        # a large window advanced with FP64 deviations
        {"name": "advance_fp64_128", "path": "advance", "precision": "fp64", "n": 128, "kind": "passive",
         "subsamples": 4, "steps": 60, "collision": "bgk"},
        # the permeability campaign: 24 uneven windows stepped together, K read now and then
        {"name": "batch24_fp32", "path": "batch", "precision": "fp32", "windows": 24, "edge": 0, "subsamples": 4,
         "steps": 20, "collision": "bgk"},
        # screening runs in 16-bit storage
        {"name": "batch8_fp16", "path": "batch", "precision": "fp16", "windows": 8, "edge": 96, "subsamples": 4,
         "steps": 20, "collision": "bgk"},
        # many fixed windows driven step by step from the host: particles in, loads and diagnostics out
        {"name": "report24_fp32", "path": "report", "precision": "fp32", "windows": 24, "edge": 0, "subsamples": 4,
         "steps": 1, "moving": False},
        # the same with particles that move, so every call rebuilds every window's geometry
        {"name": "report6_moving_fp32", "path": "report", "precision": "fp32", "windows": 6, "edge": 64,
         "subsamples": 3, "steps": 2, "moving": True},
        # d(permeability)/d(particle centres and radii): forward and backward
        {"name": "adjoint_fp32_96", "path": "adjoint", "precision": "fp32", "n": 96, "fines": 64, "subsamples": 4,
         "steps": 100, "every": 50},
        # the older coupled loop's drag proxy: voxelise, then the bounce-back solver
        {"name": "voxel_64", "path": "voxel", "n": 64, "spheres": 40, "steps": 200},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(("probe", "probe", "coupled", "converge", "advance", "batch", "batch", "report", "adjoint",
                       "voxel"))
    kind = rng.choice(KINDS)
    if path == "probe":
        return {"path": path, "precision": rng.choice(("fp64-exact", "fp64-exact", "fp32", "fp64")),
                "n": _log_int(rng, 20, 128), "kind": kind, "subsamples": rng.randint(2, 4),
                "steps": rng.randint(20, 60)}
    if path == "coupled":
        return {"path": path, "precision": rng.choice(("fp64-exact", "fp32")), "n": _log_int(rng, 20, 96),
                "kind": kind, "subsamples": rng.randint(2, 4), "steps": rng.randint(2, 10)}
    if path == "converge":
        return {"path": path, "precision": rng.choice(("fp64-exact", "fp64")), "n": _log_int(rng, 20, 96),
                "kind": kind, "subsamples": rng.randint(2, 4), "steps": rng.randint(20, 60),
                "check_every": rng.choice((1, 1, 10))}
    if path == "advance":
        return {"path": path, "precision": rng.choice(("fp64-exact", "fp64", "fp64")), "n": _log_int(rng, 32, 144),
                "kind": kind, "subsamples": rng.randint(2, 4), "steps": rng.randint(20, 60),
                "collision": "bgk"}
    if path == "batch":
        return {"path": path, "precision": rng.choice(("fp32", "fp32", "fp16", "bf16", "fp64")),
                "windows": rng.randint(2, 12), "edge": _log_int(rng, 24, 112), "subsamples": rng.randint(2, 4),
                "steps": rng.randint(10, 40), "collision": rng.choice(("bgk", "bgk", "trt"))}
    if path == "report":
        return {"path": path, "precision": rng.choice(("fp32", "fp32", "fp64-exact")),
                "windows": rng.randint(2, 12), "edge": _log_int(rng, 24, 96), "subsamples": rng.randint(2, 4),
                "steps": rng.randint(1, 5), "moving": rng.random() < 0.5}
    if path == "adjoint":
        return {"path": path, "precision": rng.choice(("fp32", "fp32", "fp64")), "n": _log_int(rng, 24, 80),
                "fines": rng.randint(8, 64), "subsamples": rng.randint(2, 4), "steps": rng.randint(30, 100),
                "every": rng.randint(20, 50)}
    return {"path": path, "n": _log_int(rng, 24, 80), "spheres": rng.randint(10, 60), "steps": rng.randint(50, 250)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _packing(kind, rng, fines_fraction=0.05, fines=None):
    """Unit-box centres, radii and the fine flag of one packing (windows.make_window's three classes)."""
    skel, r = fcc_skeleton(1.0, rng)
    c, rad, fine = [skel], [np.full(len(skel), r)], [np.zeros(len(skel), bool)]
    if kind != "skeleton":
        rf = 0.15 * r
        target = fines_fraction if fines is None else fines * 4.0 / 3.0 * np.pi * rf ** 3
        f = rsa_fines(1.0, skel, r, rf, target, rng)
        if fines is not None:
            f = f[:fines]
        if kind == "preloaded":
            f = preload(1.0, f, skel, r, rf, rng)
        c.append(f)
        rad.append(np.full(len(f), rf))
        fine.append(np.ones(len(f), bool))
    return np.vstack(c), np.concatenate(rad), np.concatenate(fine)


def _images(c, r, n, count):
    """The `count` spheres and periodic images that reach furthest into [0, n)^3 (all that enter it are among
    them), in the order of their originals, with the index of the original."""
    shifts = np.array(list(itertools.product((-1, 0, 1), repeat=3)), float) * n
    p = (c[:, None, :] + shifts[None]).reshape(-1, 3)
    rad, own = np.repeat(r, 27), np.repeat(np.arange(len(c)), 27)
    reach = rad - np.maximum(np.maximum(-p, p - n), 0.0).max(axis=1)
    keep = np.sort(np.argsort(-reach, kind="stable")[:count])
    return p[keep], rad[keep], own[keep]


def _window(n, packing, rng, moving=False):
    """(P, 10) particles of one window of edge n: the packing shifted, its axes permuted, scaled, with images."""
    c, r, fine = packing
    c = ((c + rng.uniform(0.0, 1.0, 3)) % 1.0)[:, rng.permutation(3)] * n
    k = int((~fine).sum())
    parts = [_images(c[:k], r[:k] * n, n, 4 * k)]
    if k < len(c):
        p, rad, own = _images(c[k:], r[k:] * n, n, (len(c) - k) * 27 // 20)
        parts.append((p, rad, own + k))
    p, rad, own = (np.concatenate(x) for x in zip(*parts))
    out = np.zeros((len(p), 10))
    out[:, 0:3] = p
    out[:, 3] = rad
    if moving:  # the fines drift and spin, the skeleton stands
        v = np.where(fine[:, None], rng.normal(0.0, 2.0e-4, (len(c), 3)), 0.0)
        w = np.where(fine[:, None], rng.normal(0.0, 2.0e-5, (len(c), 3)), 0.0)
        if not fine.any():
            v = rng.normal(0.0, 2.0e-4, (len(c), 3))
        out[:, 4:7] = v[own]
        out[:, 7:10] = w[own]
    return out


def _edges(case, rng):
    """Edges of a batch: the benchmark's uneven set (edge 0), or sizes around `edge`."""
    k = case["windows"]
    if case["edge"] == 0:
        return list(np.resize(BATCH_EDGES, k))
    e = case["edge"]
    lo = max(16, int(e * 0.6))
    got = [int(v) for v in np.linspace(lo, e, k).round()]
    return [v + v % 2 for v in got] if e % 2 == 0 else got


def _batch_windows(case, seed):
    rng = np.random.default_rng([seed, 17])
    packs = [_packing(k, rng) for k in KINDS]
    moving = bool(case.get("moving"))
    return [(n, _window(n, packs[i % 3], rng, moving)) for i, n in enumerate(_edges(case, rng))]


def _tau_force(case):
    """The probe's and the coupled driver's numbers along z; the benchmark's along x for batches."""
    if case["path"] in ("batch", "report"):
        return 0.8, (1.0e-6, 0.0, 0.0)
    if case["path"] == "adjoint":
        return 0.8, (1.0e-6, 0.0, 0.0)
    return 0.72, (0.0, 0.0, 2.0e-7)


def _single(case, seed):
    rng = np.random.default_rng([seed, 23])
    return _window(case["n"], _packing(case["kind"], rng), rng, case["path"] in ("coupled",))


def _moved(parts, k):
    """Where the particles are at the k-th macro step: along their velocities, to and fro."""
    out = parts.copy()
    out[:, 0:3] += parts[:, 4:7] * (100.0 if k % 2 else 200.0)
    return out


def _voxel_input(case, seed):
    rng = np.random.default_rng([seed, 29])
    pts = rng.uniform(-0.5, 0.5, (case["spheres"], 3))
    return {"points": pts, "center": np.zeros(3), "size": np.ones(3), "radius": 0.11}


def _adjoint_input(case, seed):
    rng = np.random.default_rng([seed, 31])
    p = _window(case["n"], _packing("preloaded", rng, fines=case["fines"]), rng)
    t = torch.float64 if case["precision"] == "fp64" else torch.float32
    return torch.from_numpy(p[:, 0:3].copy()).to("cuda", t), torch.from_numpy(p[:, 3].copy()).to("cuda", t)


def prepare(case, seed):
    path = case["path"]
    tau, force = _tau_force(case)
    if path in ("probe", "advance", "converge", "coupled"):
        parts = _single(case, seed)
        given = parts
        if path == "coupled":
            given = [Particle3D(*row) for row in parts.tolist()]
        more = {"collision": case["collision"]} if "collision" in case else {}
        s = SparsePscD3Q19(case["n"], given, tau=tau, subsamples=case["subsamples"], body_force_z=force[2],
                           static_geometry=path != "coupled", precision=case["precision"], **more)
        if path != "coupled":
            s.rebuild_geometry()
        scale = coupling.apply_si_scaling(case["n"], tau)
        return {"case": case, "solver": s, "parts": parts, "scale": scale, "k": 0}
    if path == "batch":
        specs = [WindowSpec(n, p, tau, force, case["subsamples"], collision=case["collision"])
                 for n, p in _batch_windows(case, seed)]
        b = PscBatch(specs, precision=case["precision"], graph_steps=10)
        b.prepare()
        return {"case": case, "batch": b}
    if path == "report":
        wins = _batch_windows(case, seed)
        cfgs = [make_config((n,) * 3, tau=tau, force=force, subsamples=case["subsamples"],
                            store=store_mode(case["precision"]), static_geometry=not case["moving"])
                for n, _ in wins]
        b = BatchHandle(cfgs)
        sets = [[_moved(p, k) if case["moving"] else p for _, p in wins] for k in range(2)]
        return {"case": case, "batch": b, "sets": sets, "k": 0}
    if path == "adjoint":
        c, r = _adjoint_input(case, seed)
        problem = PermeabilityProblem(case["n"], tau=tau, force=force, subsamples=case["subsamples"],
                                      steps=case["steps"], checkpoint_every=case["every"],
                                      precision=case["precision"])
        return {"case": case, "problem": problem, "centres": c.requires_grad_(True), "radii": r.requires_grad_(True)}
    return {"case": case, **_voxel_input(case, seed)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _as_computed(case, x):
    """A 32-bit solver's results as 32-bit numbers."""
    x = np.asarray(x)
    return x.astype(np.float32) if case["precision"] in ("fp32", "fp16", "bf16") else x


def _solver_results(case, s, diag):
    return {"diag": {k: _as_computed(case, diag[k]) for k in DIAG},
            "forces": _as_computed(case, s.hydro_forces), "torques": _as_computed(case, s.hydro_torques),
            "uz": _as_computed(case, s.uz)}


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "probe":
        s = state["solver"]
        for _ in range(case["steps"]):
            diag = s.collide_stream_psc()
        return _solver_results(case, s, diag)
    if path == "advance":
        s = state["solver"]
        return _solver_results(case, s, s.advance(case["steps"]))
    if path == "coupled":
        s = state["solver"]
        for p, x in zip(s.particles, _moved(state["parts"], state["k"])[:, 0:3].tolist()):
            p.x, p.y, p.z = x
        state["k"] += 1
        _, _, _, diag = coupling.lbm_transient_advance(s, case["steps"])
        f, t = coupling.loads_to_si(s, state["scale"]["force_scale_N_per_lu"], state["scale"]["torque_scale_Nm_per_lu"])
        out = _solver_results(case, s, diag)
        out["force_si"], out["torque_si"] = _as_computed(case, f), _as_computed(case, t)
        return out
    if path == "converge":
        s = state["solver"]
        it, residual, _, diag = coupling.lbm_converge(s, residual_tol=0.0, min_steps=1, max_steps=case["steps"],
                                                      check_every=case["check_every"])
        out = _solver_results(case, s, diag)
        out["iterations"], out["residual"] = it, residual
        return out
    if path == "batch":
        b = state["batch"]
        b.run(case["steps"])
        f = [w.f[b.parity] for w in b.windows]
        if case["precision"] in ("fp16", "bf16"):
            return f
        return [_as_computed(case, b.permeability()), f]
    if path == "report":
        b = state["batch"]
        b.set_particles_all(state["sets"][state["k"] % 2])
        state["k"] += 1
        st = b.step(case["steps"], nat.RUN_DIAG)
        d = [st[k].diag for k in range(b.nwin)]
        loads = [b.loads(k) for k in range(b.nwin)]
        return {"diag": {name: _as_computed(case, [getattr(x, name) for x in d]) for name in BATCH_DIAG},
                "forces": _as_computed(case, np.concatenate([f for f, _ in loads])),
                "torques": _as_computed(case, np.concatenate([t for _, t in loads]))}
    if path == "adjoint":
        c, r = state["centres"], state["radii"]
        c.grad = r.grad = None
        K = permeability(c, r, state["problem"])
        K.backward()
        return {"K": K.detach().to(c.dtype), "centres": c.grad, "radii": r.grad}
    solid, dx = voxel_lbm.voxelize(state["points"], state["center"], state["size"], state["radius"], case["n"])
    res = voxel_lbm.run_lbm(solid, 0.8, 1.0e-6, case["steps"], return_fields=True)
    res["solid"] = solid
    res["dx"] = dx
    return res


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_BYTES = {"fp64-exact": 8, "fp64": 8, "fp32": 4, "fp16": 2, "bf16": 2}
_FLOPS = 400.0  # arithmetic operations of one lattice update


def work(case):
    path = case["path"]
    if path == "voxel":
        n = case["n"] ** 3
        return {"bytes": case["steps"] * n * (2 * 19 * 8 + 1) + n * (4 * 8 + 1), "flops": case["steps"] * n * _FLOPS}
    s = _BYTES[case["precision"]]
    solid = 8 if case["precision"] == "fp64-exact" else 1
    if path == "adjoint":
        n = case["n"] ** 3
        # forward, the reverse step (state, adjoint in and out) and the forward states it needs again
        return {"bytes": case["steps"] * n * (2 * (2 * 19 * s + 8) + 3 * 19 * s + 8), "flops": case["steps"] * n * 4 * _FLOPS}
    if path in ("batch", "report"):
        n = float(sum(int(e) ** 3 for e in _edges(case, None)))
    else:
        n = float(case["n"] ** 3)
    return {"bytes": case["steps"] * n * (2 * 19 * s + solid), "flops": case["steps"] * n * _FLOPS}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------
_C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
      (1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1),
      (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
_W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _opp(i):
    return 0 if i == 0 else (i + 1 if i % 2 else i - 1)


def _box(p, n):
    lo = [max(0, math.floor(p[a] - p[3] - 1.0)) for a in range(3)]
    hi = [min(n, math.ceil(p[a] + p[3] + 1.0)) for a in range(3)]
    return None if any(h <= l for l, h in zip(lo, hi)) else list(zip(lo, hi))


def _samples(lo, hi, S, c, dev):
    o = (torch.arange(S, dtype=torch.float64, device=dev) + 0.5) / S
    return (torch.arange(lo, hi, dtype=torch.float64, device=dev)[:, None] + o[None]).reshape(-1) - c


def _voxelise(n, parts, S):
    """alpha_sum, the particles' own fractions on their boxes, and the solid velocity (None: all stand)."""
    dev = _dev()
    total = torch.zeros((n, n, n), dtype=torch.float64, device=dev)
    moving = bool(np.any(parts[:, 4:10]))
    us = torch.zeros((3, n, n, n), dtype=torch.float64, device=dev) if moving else None
    own = []
    for p in parts:
        b = _box(p, n)
        if b is None:
            own.append(None)
            continue
        d = [_samples(l, h, S, float(p[a]), dev) ** 2 for a, (l, h) in enumerate(b)]
        e = [h - l for l, h in b]
        inside = ((d[0][:, None] + d[1][None])[:, :, None] + d[2]) <= float(p[3]) * float(p[3])
        a = inside.view(e[0], S, e[1], S, e[2], S).sum((1, 3, 5)).double() / S ** 3
        sl = tuple(slice(l, h) for l, h in b)
        total[sl] += a
        own.append((sl, a))
        if moving:
            r = _arms(p, b, dev)
            for k in range(3):
                u, v = (k + 1) % 3, (k + 2) % 3
                us[(k, *sl)] += a * (float(p[4 + k]) + float(p[7 + u]) * r[v] - float(p[7 + v]) * r[u])
    if moving:
        us = torch.where(total > 1e-14, us / total.clamp_min(1e-14), us)
    return total, own, us


def _arms(p, b, dev):
    return [(torch.arange(l, h, dtype=torch.float64, device=dev) + 0.5 - float(p[a])).view([-1 if k == a else 1 for k in range(3)])
            for a, (l, h) in enumerate(b)]


def _pull_moments(g, F):
    drho = g.sum(0)
    rho = 1.0 + drho
    m = [sum(c[a] * g[i] for i, c in enumerate(_C) if c[a]) for a in range(3)]
    return drho, rho, m, [(m[a] + 0.5 * F[a]) / rho for a in range(3)]


def _collide(g, solid, us, tau, taum, F):
    """Post-collision deviations f - w and the node momentum of the solid term."""
    drho, rho, m, _ = _pull_moments(g, F)
    u = [(m[a] + F[a]) / rho for a in range(3)]
    uu = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    B = solid / (solid + tau * (1.0 - solid) + 1e-14)

    def eq(c, w, v, vv):
        cu = c[0] * v[0] + c[1] * v[1] + c[2] * v[2]
        return w * (drho + rho * (3.0 * cu + 4.5 * cu * cu - 1.5 * vv))

    uF = sum(u[a] * F[a] for a in range(3))
    geq = [eq(c, w, u, uu) for c, w in zip(_C, _W)]
    if us is not None:
        vv = us[0] ** 2 + us[1] ** 2 + us[2] ** 2
    out, imb = [], [0.0, 0.0, 0.0]
    for i, (c, w) in enumerate(zip(_C, _W)):
        j = _opp(i)
        gs = w * drho if us is None else eq(c, w, us, vv)
        bos = B * (g[j] - g[i] + gs - geq[j])
        cF = sum(c[a] * F[a] for a in range(3))
        cu = sum(c[a] * u[a] for a in range(3)) if i else 0.0
        guo = (1.0 - 0.5 / tau) * w * (9.0 * cu * cF - 3.0 * uF) + (1.0 - 0.5 / taum) * w * 3.0 * cF
        if taum == tau:
            relax = (g[i] - geq[i]) / tau
        else:
            relax = 0.5 * ((g[i] + g[j] - geq[i] - geq[j]) / tau + (g[i] - g[j] - geq[i] + geq[j]) / taum)
        out.append(g[i] - (1.0 - B) * relax + bos + guo)
        for a in range(3):
            if c[a]:
                imb[a] = imb[a] + c[a] * bos
    return torch.stack(out), imb


def _stream(g):
    return torch.stack([torch.roll(g[i], c, (0, 1, 2)) if any(c) else g[i] for i, c in enumerate(_C)])


def _loads(parts, own, total, imb):
    F, T = np.zeros((len(parts), 3)), np.zeros((len(parts), 3))
    dev = total.device
    rows = []
    for p, o in zip(parts, own):
        if o is None:
            rows.append(torch.zeros(6, dtype=torch.float64, device=dev))
            continue
        sl, a = o
        w = a / total[sl].clamp_min(1e-14)
        f = [-(w * imb[k][sl]) for k in range(3)]
        r = _arms(p, [(s.start, s.stop) for s in sl], dev)
        t = [r[1] * f[2] - r[2] * f[1], r[2] * f[0] - r[0] * f[2], r[0] * f[1] - r[1] * f[0]]
        rows.append(torch.stack([x.sum() for x in f + t]))
    if rows:
        x = torch.stack(rows).cpu().numpy()
        F, T = x[:, 0:3].copy(), x[:, 3:6].copy()
    return F, T


def _advance(n, parts, S, tau, taum, F, steps, g=None, geometry=None):
    """`steps` collide-stream steps; the streamed deviations, the unstreamed ones, the last node momentum, the
    geometry, and mean u_z after every step."""
    geometry = geometry or _voxelise(n, parts, S)
    total, own, us = geometry
    solid = total.clamp(0.0, 1.0)
    if g is None:
        g = torch.zeros((19, n, n, n), dtype=torch.float64, device=total.device)
    means = []
    for _ in range(steps):
        post, imb = _collide(g, solid, us, tau, taum, F)
        g = _stream(post)
        means.append(_pull_moments(g, F)[3][2].mean())
    return g, post, imb, geometry, [float(x) for x in means]


def _exact_solver(case, seed):
    tau, F = _tau_force(case)
    parts = _single(case, seed)
    if case["path"] == "coupled":
        parts = _moved(parts, 0)
    g, _, imb, (total, own, _), means = _advance(case["n"], parts, case["subsamples"], tau, tau, F, case["steps"])
    f, t = _loads(parts, own, total, imb)
    norm = lambda v: float(np.sqrt((v * v).sum(1)).max()) if len(v) else 0.0  # noqa: E731
    uz = _pull_moments(g, F)[3][2]
    out = {"diag": dict(zip(DIAG, (float(total.clamp(0.0, 1.0).sum()), means[-1], norm(f), norm(t)))), "forces": f,
           "torques": t, "uz": uz}
    if case["path"] == "coupled":
        scale = coupling_scales(case["n"], tau)
        out["force_si"], out["torque_si"] = scale[0] * f, scale[1] * t
    if case["path"] == "converge":
        out["iterations"] = None
        out["residual"] = abs(means[-1] - means[-2]) / max(abs(means[-1]), 1e-30)
    return out


def coupling_scales(n, tau, temperature=773.15, pressure=2.0e5, mu=3.7e-5, box=0.009):
    """Force and torque scales of helium at (T, p), lattice units to SI."""
    rho = pressure / (2077.1 * temperature)
    dx = box / n
    dt = (tau - 0.5) / 3.0 * dx * dx / (mu / rho)
    return rho * dx ** 4 / dt ** 2, rho * dx ** 5 / dt ** 2


def _darcy(g, solid, tau, F):
    u = _pull_moments(g, F)[3]
    fmag = math.sqrt(sum(x * x for x in F))
    flux = sum(((1.0 - solid) * u[a]).sum() * (F[a] / fmag) for a in range(3))
    return (tau - 0.5) / 3.0 * flux / g[0].numel() / fmag


def _exact_batch(case, seed):
    tau, F = _tau_force(case)
    taum = trt_tau_minus_of(tau) if case.get("collision") == "trt" else tau
    K, fields, diag, forces, torques = [], [], [], [], []
    scale = 2.0 ** 20 if case["precision"] == "fp16" else 1.0
    report = case["path"] == "report"
    if report:
        steps = case["steps"]
    else:  # the batch takes one step while it is prepared
        steps = case["steps"] + 1
    for n, parts in _batch_windows(case, seed):
        if report and case["moving"]:
            parts = _moved(parts, 0)
        g, post, imb, (total, own, _), means = _advance(n, parts, case["subsamples"], tau, taum, F, steps)
        solid = total.clamp(0.0, 1.0)
        K.append(float(_darcy(g, solid, tau, F)))
        if report:
            f, t = _loads(parts, own, total, imb)
            norm = lambda v: float(np.sqrt((v * v).sum(1)).max()) if len(v) else 0.0  # noqa: E731
            diag.append([float(solid.sum()), norm(f), norm(t), K[-1], float((1.0 - solid).sum())])
            forces.append(f)
            torques.append(t)
        else:
            fields.append((post * scale).reshape(-1))
    if report:
        return {"diag": dict(zip(BATCH_DIAG, np.array(diag).T.copy())), "forces": np.concatenate(forces), "torques": np.concatenate(torques)}
    return fields if case["precision"] in ("fp16", "bf16") else [np.array(K), fields]


def trt_tau_minus_of(tau, magic=3.0 / 16.0):
    return 0.5 + magic / (tau - 0.5)


def _smooth_box(c, r, b, S, eps, dev):
    o = (torch.arange(S, dtype=torch.float64, device=dev) + 0.5) / S
    x = [((torch.arange(l, h, dtype=torch.float64, device=dev)[:, None] + o[None]).reshape(-1) - c[a]) ** 2
         for a, (l, h) in enumerate(b)]
    d = ((x[0][:, None] + x[1][None])[:, :, None] + x[2]).clamp_min(1e-24).sqrt()
    e = [h - l for l, h in b]
    s = 0.5 * (1.0 + torch.tanh(0.5 * (r - d) / eps))
    return s.view(e[0], S, e[1], S, e[2], S).mean((1, 3, 5))


def _exact_adjoint(case, seed):
    tau, F = _tau_force(case)
    n, S, eps = case["n"], case["subsamples"], 0.05
    c, r = (x.double().to(_dev()) for x in _adjoint_input(case, seed))
    rows = torch.cat([c, r[:, None]], 1).cpu().numpy()
    boxes = [_box(p, n) for p in rows]
    total = torch.zeros((n, n, n), dtype=torch.float64, device=c.device)
    for k, b in enumerate(boxes):
        if b is not None:
            total[tuple(slice(l, h) for l, h in b)] += _smooth_box(c[k], r[k], b, S, eps, c.device)
    total.requires_grad_(True)
    solid = total.clamp(0.0, 1.0)

    def some(g, s, k):
        for _ in range(k):
            g = _stream(_collide(g, s, None, tau, tau, F)[0])
        return g

    g = torch.zeros((19, n, n, n), dtype=torch.float64, device=c.device)
    done = 0
    while done < case["steps"]:
        k = min(4, case["steps"] - done)
        g = torch.utils.checkpoint.checkpoint(some, g, solid, k, use_reentrant=False)
        done += k
    K = _darcy(g, solid, tau, F)
    K.backward()
    gc, gr = torch.zeros_like(c), torch.zeros_like(r)
    for k, b in enumerate(boxes):
        if b is None:
            continue
        x, y = c[k].clone().requires_grad_(True), r[k].clone().requires_grad_(True)
        (_smooth_box(x, y, b, S, eps, c.device) * total.grad[tuple(slice(l, h) for l, h in b)]).sum().backward()
        gc[k], gr[k] = x.grad, y.grad
    return {"K": K.detach(), "centres": gc, "radii": gr}


def _exact_voxel(case, seed):
    n, tau, fz = case["n"], 0.8, 1.0e-6
    v = _voxel_input(case, seed)
    dev = _dev()
    lo = v["center"] - 0.5 * v["size"]
    dx = v["size"] / n
    ax = [torch.from_numpy(lo[a] + (np.arange(n) + 0.5) * dx[a]).to(dev) for a in range(3)]
    solid = torch.zeros((n, n, n), dtype=torch.bool, device=dev)
    for p in v["points"]:
        d = [(ax[a] - float(p[a])) ** 2 for a in range(3)]
        solid |= ((d[0][:, None] + d[1][None])[:, :, None] + d[2]) <= v["radius"] * v["radius"]
    F = (0.0, 0.0, fz)
    w = torch.tensor(_W, dtype=torch.float64, device=dev)
    g = torch.zeros((19, n, n, n), dtype=torch.float64, device=dev)

    def moments(g):
        drho, rho, _, u = _pull_moments(g, F)
        return drho, rho, [torch.where(solid, torch.zeros_like(x), x) for x in u]

    for _ in range(case["steps"]):
        drho, rho, u = moments(g)
        uu = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        uF = u[2] * fz
        out = []
        for i, c in enumerate(_C):
            cu = c[0] * u[0] + c[1] * u[1] + c[2] * u[2]
            eq = w[i] * (drho + rho * (3.0 * cu + 4.5 * cu * cu - 1.5 * uu))
            guo = (1.0 - 0.5 / tau) * w[i] * (3.0 * (c[2] * fz - uF) + 9.0 * cu * c[2] * fz)
            out.append(g[i] - (g[i] - eq) / tau + guo)
        g = _stream(torch.stack(out))
        for k in range(9):  # the solver's own overwrite of each pair at solid nodes
            g[2 * k + 1] = torch.where(solid, g[2 * k + 2], g[2 * k + 1])
    _, _, u = moments(g)
    fluid = ~solid
    uz = u[2]
    nu = (tau - 0.5) / 3.0
    return {"mean_uz_fluid": float(uz[fluid].mean()), "superficial_uz": float(uz.mean()), "max_uz": float(uz[fluid].max()),
            "permeability_lu": nu * float(uz.mean()) / fz, "porosity_voxel": float(fluid.double().mean()),
            "speed_slice": uz[:, :, n // 2], "solid_slice": None, "ux": u[0], "uy": u[1], "uz": uz, "solid": None,
            "dx": dx}


def exact(case, seed):
    path = case["path"]
    with torch.no_grad() if path != "adjoint" else torch.enable_grad():
        if path in ("probe", "advance", "converge", "coupled"):
            return _exact_solver(case, seed)
        if path in ("batch", "report"):
            return _exact_batch(case, seed)
        if path == "adjoint":
            return _exact_adjoint(case, seed)
        return _exact_voxel(case, seed)
