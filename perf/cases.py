"""Workloads of the N-body engine, each through the entry points that a
program calls: the force-backend seam on host arrays, the integrator seam,
device-resident stepping with a read-back per frame, batched ensembles and the
energy diagnostics.  Sizes are those of the benchmark's configurations and
ragged ones between them; all inputs come from the seeded scene generators.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "celestial-mechanics-desktop_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from nbody_b200 import scenarios  # noqa: E402

EPS = 1e-4
STATE = ("px", "py", "pz", "vx", "vy", "vz", "ax", "ay", "az", "mass", "radius", "active")
# the disk's radii grow by this much, so that about 1 % of the bodies merge per 1000 steps
DISK_RADIUS_SCALE = 30.0
# bodies of the sphere that the learned criterion is trained on, and its error budget (log10)
TRAIN_N, MAC_BUDGET = 65536, -3.18


def _forces(n, mode, **kw):
    return {"kind": "forces", "n": n, "mode": mode, "theta": 0.5, "shell": False, "quad": True,
            "eps": EPS, **kw}


def _steps(n, mode, steps, dt, **kw):
    return {"kind": "steps", "n": n, "mode": mode, "steps": steps, "dt": dt, "theta": 0.5,
            "learned": False, "yoshida": False, "eps": EPS, **kw}


def listed():
    return [
        # The smallest call: one force evaluation of a desktop scene through the backend seam, in
        # the CPU backend's own arithmetic.  Launches and latency count.
        {"name": "forces_fp64_1k", **_forces(1000, "fp64")},
        # An interactive Barnes-Hut scene of an odd size, one evaluation per call.
        {"name": "forces_bh_20k", **_forces(20011, "bh")},
        # The largest call at the seam: host arrays of 2^20 bodies in, accelerations out.
        {"name": "forces_bh_1m", **_forces(1 << 20, "bh")},
        # The FP32 direct sum of a mid-sized ragged scene (when a tree's error is not wanted).
        {"name": "forces_direct_100k", **_forces(100003, "direct")},
        # The desktop app's own Barnes-Hut semantics (per-body criterion, monopoles, FP64).
        {"name": "forces_ref_50k", **_forces(50021, "bh_ref")},
        # A small cluster integrated on the device in FP64, read back after a thousand steps.
        {"name": "steps_fp64_1k", **_steps(1000, "fp64", 1000, 1e-3)},
        # The integrator seam: a BodySoA goes up, ten steps run, the BodySoA comes back.
        {"name": "integrate_bh_100k", "kind": "integrate", "n": 100003, "mode": "bh", "steps": 10,
         "dt": 1e-4, "theta": 0.5, "shell": False, "quad": True, "eps": EPS},
        # The Barnes-Hut configuration of 2^20 bodies: a frame of twenty steps, read back.
        {"name": "steps_bh_1m", **_steps(1 << 20, "bh", 20, 1e-4)},
        # The same sphere and frame under the learned opening criterion, with its audit.
        {"name": "steps_learned_1m", **_steps(1 << 20, "bh", 20, 1e-4, learned=True)},
        # The collisional disk: shell theorem, broad phase, merges and compaction every step.
        {"name": "disk_262k", "kind": "disk", "n": 262144, "steps": 50, "dt": 1e-3},
        # 512 independent systems of 64 to 8192 bodies, stepped together and read back.
        {"name": "ensemble_512", "kind": "ensemble", "systems": 512, "sizes_seed": 3, "steps": 20,
         "dt": 1e-4},
        # The energy and momentum read-out that a run logs beside its frames, exact potential.
        {"name": "energy_64k", "kind": "energy", "n": 65537, "pe_mode": 0},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forces"] * 5 + ["steps"] * 3 + ["integrate", "disk", "ensemble", "energy"])
    eps = rng.choice([EPS, EPS, 1e-2])
    theta = rng.choice([0.5, 0.5, 0.7, 0.9])
    if kind == "forces":
        mode = rng.choice(["fp64", "bh", "bh", "direct", "bh_ref"])
        n = _size(rng, *{"fp64": (200, 8192), "bh": (4000, 1 << 20), "direct": (2000, 131072),
                         "bh_ref": (2000, 65536)}[mode])
        return _forces(n, mode, theta=theta, eps=rng.choice([eps, 0.0]),
                       shell=rng.random() < 0.2,
                       quad=not (mode == "bh" and rng.random() < 0.2))
    if kind == "steps":
        mode = rng.choice(["fp64", "bh", "learned"])
        if mode == "fp64":
            return _steps(_size(rng, 200, 4096), "fp64", rng.randrange(100, 400), 1e-3, eps=eps,
                          yoshida=rng.random() < 0.3)
        if mode == "bh":
            return _steps(_size(rng, 8000, 1 << 20), "bh", rng.randrange(5, 21), 1e-4, eps=eps,
                          theta=theta)
        return _steps(_size(rng, 65536, 1 << 20), "bh", rng.randrange(5, 21), 1e-4, learned=True)
    if kind == "integrate":
        return {"kind": kind, "n": _size(rng, 2000, 400000), "mode": "bh",
                "steps": rng.randrange(1, 11), "dt": 1e-4, "theta": theta,
                "shell": rng.random() < 0.3, "quad": True, "eps": eps}
    if kind == "disk":
        return {"kind": kind, "n": _size(rng, 20000, 262144), "steps": rng.randrange(5, 51),
                "dt": 1e-3}
    if kind == "ensemble":
        return {"kind": kind, "systems": _size(rng, 32, 512), "sizes_seed": rng.randrange(1000),
                "steps": rng.randrange(5, 21), "dt": 1e-4}
    pe_mode = rng.randrange(2)
    return {"kind": "energy", "n": _size(rng, 2000, (1 << 20) if pe_mode else 131072),
            "pe_mode": pe_mode}


def _scene(case, seed):
    """The bodies of a case, from its seed alone."""
    if case["kind"] == "disk":
        return scenarios.collisional_disk(case["n"], seed=seed, radius_scale=DISK_RADIUS_SCALE)
    return scenarios.plummer(case["n"], seed=seed)


def _systems(case, seed):
    sizes = scenarios.ensemble_sizes(case["systems"], seed=case["sizes_seed"])
    return sizes, [scenarios.plummer(int(k), seed=seed * 100003 + s) for s, k in enumerate(sizes)]


def _backend(case):
    import nbody_b200 as nb

    modes = {"fp64": nb.MODE_DIRECT_FP64, "direct": nb.MODE_DIRECT, "bh": nb.MODE_BARNES_HUT,
             "bh_ref": nb.MODE_BARNES_HUT_REF}
    be = nb.B200PhysicsBackend(case["n"], modes[case["mode"]], theta=case["theta"])
    be.enable_shell_theorem, be.use_quadrupole = case.get("shell", False), case.get("quad", True)
    return be


def _train(e, nb):
    """The learned criterion's network, trained on a smaller sphere as a user would."""
    e.set_state(scenarios.plummer(min(TRAIN_N, e.capacity), seed=10), old_acc=False)
    e.step(1, 0.0, EPS, nb.MODE_BARNES_HUT)
    e.mac_harvest(2_000_000, 0.5, 10, EPS)
    e.mac_train(3, 4096, 2e-3, seed=3)


def prepare(case, seed):
    import nbody_b200 as nb

    kind = case["kind"]
    if kind == "ensemble":
        sizes, systems = _systems(case, seed)
        ens = nb.Ensemble(sizes)
        # what the autotuners keep on this distribution of sizes, set by hand
        # so that every process runs the same plan
        ens.set_param(nb.native.PARAM_ENS_DIRECT_SHAPE, 0)
        ens.set_param(nb.native.PARAM_GROUP_SPAN, 512)
        ens.set_param(nb.native.PARAM_GROUP_BODIES, 64)
        ens.set_state(systems)
        ens.compute_forces(EPS)
        return {"case": case, "ens": ens}
    bodies = _scene(case, seed)
    if kind in ("forces", "integrate"):
        return {"case": case, "backend": _backend(case), "bodies": bodies,
                "integrator": nb.B200SoAIntegrator()}
    e = nb.Engine(bodies.n)
    if kind == "energy":
        e.set_state(bodies)
        return {"case": case, "engine": e}
    if kind == "disk":
        flags = nb.MODE_BARNES_HUT | nb.FLAG_SHELL_THEOREM | nb.FLAG_COLLISIONS
    elif case["mode"] == "fp64":
        flags = nb.MODE_DIRECT_FP64 | (nb.FLAG_YOSHIDA4 if case["yoshida"] else 0)
    else:
        flags = nb.MODE_BARNES_HUT
        e.set_param(nb.native.PARAM_THETA, float(case["theta"]))
    if case.get("learned"):
        _train(e, nb)
        e.set_param(nb.native.PARAM_MAC_BUDGET, MAC_BUDGET)
        # the criterion's error is audited against the direct sum as it runs
        e.set_param(nb.native.PARAM_MAC_AUDIT_RMS, 3e-3)
        e.set_param(nb.native.PARAM_MAC_AUDIT_INTERVAL, case["steps"])
    e.set_state(bodies, old_acc=False)
    # accelerations at the starting positions
    e.step(1, 0.0, case.get("eps", EPS), flags & ~nb.FLAG_COLLISIONS)
    if case.get("learned"):
        flags |= nb.FLAG_LEARNED_MAC
    state = {"case": case, "engine": e, "flags": flags}
    if kind == "disk":
        # the program's own frame: rows of merged bodies leave the end of it
        state["frame"] = {k: np.zeros_like(getattr(bodies, k)) for k in STATE}
        state["frame"]["ids"] = np.zeros(bodies.n, np.int32)
    return state


def _fields(bodies):
    return {k: getattr(bodies, k) for k in STATE[:9]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forces":
        b = state["bodies"]
        state["backend"].compute_forces(b, case["eps"])
        return {"ax": b.ax, "ay": b.ay, "az": b.az}
    if kind == "integrate":
        b = state["bodies"]
        state["integrator"].step(b, state["backend"], case["eps"], case["dt"], case["steps"])
        return _fields(b)
    if kind == "ensemble":
        state["ens"].step(case["steps"], case["dt"], EPS)
        return state["ens"].get_state()
    e = state["engine"]
    if kind == "energy":
        return e.diagnostics(EPS, case["pe_mode"])
    e.step(case["steps"], case["dt"], case.get("eps", EPS), state["flags"])
    b, ids = e.get_state()
    got = {**{k: getattr(b, k) for k in STATE}, "ids": ids}
    if kind != "disk":
        return got
    for k, v in got.items():
        state["frame"][k][:b.n] = v
    return {**state["frame"], "rows": b.n}


def work(case):
    """Bytes: what the call reads and writes once.  Flops: 20 per body pair of
    a direct sum; for a tree an estimate of the interactions that the opening
    angle asks for, (28 pi / 9) ln n / theta^2 per body, 51 flops each with
    quadrupoles."""
    kind = case["kind"]
    if kind == "ensemble":
        # sizes log-uniform in [64, 8192]: mean size and mean square size
        span = math.log(8192 / 64)
        n = case["systems"] * (8192 - 64) / span
        small = case["systems"] * (2048 ** 2 - 64 ** 2) / (2 * span)
        large = case["systems"] * (8192 - 2048) / span
        per = 51 * (28 * math.pi / 9) * math.log(5000) / 0.25
        return {"bytes": 56.0 * n + 72.0 * n, "flops": case["steps"] * (20 * small + per * large)}
    n = case["n"]
    pairs = float(n) * n
    theta = case.get("theta", 0.5)
    per = 51 if case.get("quad", True) and case.get("mode") != "bh_ref" else 20
    tree = per * n * (28 * math.pi / 9) * math.log(n) / theta ** 2
    if kind == "energy":
        return {"bytes": 73.0 * n, "flops": 40.0 * n + (tree if case["pe_mode"] else 6 * pairs)}
    one = tree if case.get("mode", "bh") in ("bh", "bh_ref") else 20 * pairs
    if kind == "forces":
        return {"bytes": 33.0 * n + 24.0 * n, "flops": one}
    reps = case["steps"] * (3 if case.get("yoshida") else 1)
    return {"bytes": 81.0 * n + 93.0 * n, "flops": reps * one}


# ---- the same in 64 bits, by torch ------------------------------------------

EXACT_PAIRS = 1.5e11  # beyond this a direct sum takes too long


def _rows(bodies, keys):
    return [torch.from_numpy(np.ascontiguousarray(getattr(bodies, k), np.float64)).cuda()
            for k in keys]


def _direct(x, m, eps, radius=None):
    """Accelerations of all bodies at x (n, 3): the softened direct sum, with a
    source of radius R pulling as a softened shell inside it."""
    n = len(m)
    out = torch.empty_like(x)
    step = max(1, (1 << 26) // n)
    for i in range(0, n, step):
        d = x[i:i + step, None, :] - x[None, :, :]
        r2 = (d * d).sum(-1)
        soft = r2 + eps * eps
        w = m * torch.where(soft > 0, soft, torch.inf).pow(-1.5)
        if radius is not None:
            w = torch.where((radius > 0) & (r2 < radius * radius),
                            m * (radius * radius + eps * eps).pow(-1.5), w)
        out[i:i + step] = -(w[..., None] * d).sum(1)
    return out


def _verlet(x, v, a, m, eps, dts):
    for dt in dts:
        v = v + 0.5 * dt * a
        x = x + dt * v
        a = _direct(x, m, eps)
        v = v + 0.5 * dt * a
    return x, v, a


def _dts(case):
    dt = case["dt"]
    if not case.get("yoshida"):
        return [dt] * case["steps"]
    c = 2.0 ** (1.0 / 3.0)
    return [dt / (2.0 - c), -c * dt / (2.0 - c), dt / (2.0 - c)] * case["steps"]


def _moved(b, eps, dts, old_acc):
    x, v = (torch.stack(_rows(b, k), 1) for k in (("px", "py", "pz"), ("vx", "vy", "vz")))
    m, = _rows(b, ("mass",))
    a = _direct(x, m, eps) if old_acc else torch.zeros_like(x)
    return torch.cat(_verlet(x, v, a, m, eps, dts), 1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "disk":
        return None
    if kind == "ensemble":
        _, systems = _systems(case, seed)
        if sum(float(b.n) ** 2 for b in systems) * case["steps"] > EXACT_PAIRS:
            return None
        got = np.concatenate([_moved(b, EPS, _dts(case), True) for b in systems])
        return {k: got[:, i].copy() for i, k in enumerate(STATE[:9])}
    n = case["n"]
    if float(n) * n * case.get("steps", 1) * (3 if case.get("yoshida") else 1) > EXACT_PAIRS:
        return None
    b = _scene(case, seed)
    if kind == "forces":
        x = torch.stack(_rows(b, ("px", "py", "pz")), 1)
        m, r = _rows(b, ("mass", "radius"))
        a = _direct(x, m, case["eps"], r if case["shell"] else None).cpu().numpy()
        return {k: a[:, i].copy() for i, k in enumerate(("ax", "ay", "az"))}
    if kind == "integrate":
        if case["shell"]:
            return None
        got = _moved(b, case["eps"], _dts(case), False)
        return {k: got[:, i].copy() for i, k in enumerate(STATE[:9])}
    if kind == "steps":
        got = _moved(b, case["eps"], _dts(case), True)
        return {**{k: got[:, i].copy() for i, k in enumerate(STATE[:9])},
                **dict.fromkeys(("mass", "radius", "active", "ids"))}
    x, v = (torch.stack(_rows(b, k), 1) for k in (("px", "py", "pz"), ("vx", "vy", "vz")))
    m, = _rows(b, ("mass",))
    pe = 0.0
    step = max(1, (1 << 26) // n)
    for i in range(0, n, step):
        d = x[i:i + step, None, :] - x[None, :, :]
        inv = ((d * d).sum(-1) + EPS * EPS).rsqrt()
        inv[torch.arange(len(inv)), torch.arange(i, i + len(inv))] = 0.0
        pe -= 0.5 * float((m[i:i + step, None] * m * inv).sum())
    ke = float((0.5 * m * (v * v).sum(1)).sum())
    p, com = (m[:, None] * v).sum(0).tolist(), (m[:, None] * x).sum(0) / m.sum()
    ang = (m[:, None] * torch.linalg.cross(x, v)).sum(0).tolist()
    return {"ke": ke, "pe": pe, "e": ke + pe, **dict(zip(("px", "py", "pz"), p)),
            **dict(zip(("lx", "ly", "lz"), ang)),
            **dict(zip(("comx", "comy", "comz"), com.tolist())), "m": float(m.sum())}
