"""The calls a program makes into this framework, as cases to be timed.

A case is one pass through the public entry points: KDK steps of one system, a
force and potential evaluation with the energies, the field at probe points,
adaptive steps, or a batch of systems through the many-system engine.  State
lives on the GPU between the calls; results come back to the host through
nb_download into pinned memory, as a host program that owns the arrays takes
them.  The mixed-precision form evaluates its pairs in FP32 and widens the sums
into FP64 buffers: its accelerations and potentials are returned in 32 bits,
positions, velocities, energies and everything of the FP64 form in 64.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "astronbodysim.jl_gb300"))
import astronbodysim as nb  # noqa: E402
from astronbodysim import _lib as L  # noqa: E402

# Largest listed work of one pass, in interactions (pairs times force evaluations).
MOST_PAIRS = (1 << 20) ** 2


def listed():
    return [
        # A star cluster small enough that launches and the host decide the time.
        _step("step_1000", 1000, steps=10, eps=1e-2, dt=1e-3),
        # The framework's plain configuration: Plummer sphere, N = 4096, eps = 0.01, dt = 1e-3.
        _step("step_4096", 4096, steps=10, eps=1e-2, dt=1e-3),
        # A cluster with a mass spectrum under the Plummer law, a size that fills no tile.
        _step("step_24593_plummer_law", 24593, steps=5, eps=1e-2, dt=1e-3, law="plummer", masses="spread"),
        # A cuspy galaxy halo at the resolution of an ordinary run.
        _step("step_100003_hernquist", 100003, steps=2, eps=5e-3, dt=1e-3, model="hernquist"),
        # A large halo whose particles differ in mass.
        _step("step_400001_masses", 400001, steps=1, eps=1e-3, dt=1e-4, masses="spread"),
        # The framework's large configuration: Plummer sphere, N = 2^20, eps = 1e-3, dt = 1e-4.
        _step("step_1048576", 1 << 20, steps=1, eps=1e-3, dt=1e-4),
        # A snapshot of a running simulation: forces, potentials and energies.
        {"name": "snapshot_50021", "kind": "snapshot", "n": 50021, "model": "plummer", "masses": "equal",
         "law": "spline", "eps": 1e-2},
        # The field of a cluster on probe points: a rotation curve or a potential map.
        {"name": "probe_10007_in_30011", "kind": "probe", "n": 30011, "points": 10007, "model": "plummer",
         "masses": "equal", "law": "spline", "eps": 1e-2},
        # Two galaxies in collision with individual power-of-two time steps.
        {"name": "collision_adaptive_2x16384", "kind": "adaptive", "n_each": 16384, "steps": 12, "eps": 5e-3},
        # Many small independent systems integrated together (the ensemble: N in [64, 8192]).
        {"name": "ensemble_160", "kind": "ensemble", "systems": 160, "n_min": 64, "n_max": 8192,
         "steps_min": 40, "steps_max": 40, "sizes_seed": 3, "law": "spline"},
        # Requests of a serving stream: few systems of very uneven size, uneven step counts.
        {"name": "serving_12", "kind": "ensemble", "systems": 12, "n_min": 256, "n_max": 65536,
         "steps_min": 5, "steps_max": 15, "sizes_seed": 34, "law": "spline"},
        # The plain FP64 form, the run that a mixed-precision one is judged by.
        _step("step_4096_fp64", 4096, steps=2, eps=1e-2, dt=1e-3, precision="fp64"),
    ]


def _step(name, n, *, steps, eps, dt, model="plummer", masses="equal", law="spline", precision="mixed"):
    c = {"kind": "step", "n": n, "steps": steps, "eps": eps, "dt": dt, "model": model, "masses": masses,
         "law": law, "precision": precision}
    return dict(c, name=name) if name else c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "snapshot", "probe", "adaptive", "ensemble", "fp64"])
    eps = round(math.exp(rng.uniform(math.log(1e-3), math.log(1e-2))), 5)
    model = rng.choice(["plummer", "plummer", "hernquist"])
    masses = rng.choice(["equal", "equal", "spread"])
    law = rng.choice(["spline", "spline", "plummer"])
    if kind == "step":
        n = _log_int(rng, 1000, 1 << 20)
        steps = max(1, min(rng.randint(1, 10), MOST_PAIRS // (8 * n * n)))
        # as the configurations: 1e-3 for small and ordinary systems, 1e-4 for large ones
        return _step(None, n, steps=steps, eps=eps, dt=1e-3 if n < 200000 else 1e-4, model=model,
                     masses=masses, law=law)
    if kind == "fp64":
        return _step(None, _log_int(rng, 1000, 12000), steps=1, eps=eps, dt=1e-3, model=model, masses=masses,
                     law=law, precision="fp64")
    if kind == "snapshot":
        return {"kind": "snapshot", "n": _log_int(rng, 2000, 300000), "model": model, "masses": masses,
                "law": law, "eps": eps}
    if kind == "probe":
        return {"kind": "probe", "n": _log_int(rng, 2000, 200000), "points": _log_int(rng, 100, 50000),
                "model": model, "masses": masses, "law": law, "eps": eps}
    if kind == "adaptive":
        return {"kind": "adaptive", "n_each": _log_int(rng, 1000, 50000), "steps": rng.randint(4, 16),
                "eps": 5e-3}
    systems = _log_int(rng, 8, 256)
    steps = rng.randint(10, 40)
    return {"kind": "ensemble", "systems": systems, "n_min": 64, "n_max": 32768 if systems <= 32 else 8192,
            "steps_min": rng.randint(10, steps), "steps_max": steps, "sizes_seed": rng.randrange(1 << 20),
            "law": law}


# ---- inputs ---------------------------------------------------------------


def _cluster(case, n, seed):
    """A seeded sphere on its way through space (so its total momentum is not zero)."""
    make = nb.hernquist if case["model"] == "hernquist" else nb.plummer
    d = make(n, seed=2 * seed)
    if case["masses"] == "spread":
        d["mass"] = np.random.default_rng(2 * seed + 1).uniform(0.5, 1.5, n) / n
    d["vel"] = d["vel"] + np.array([0.1, -0.2, 0.05])
    return d


def _systems(case, seed=None):
    """(N, steps, eps) of an ensemble's systems, from the case alone; with a seed also their particles."""
    r = random.Random(case["sizes_seed"])
    got = []
    for k in range(case["systems"]):
        n, steps = _log_int(r, case["n_min"], case["n_max"]), r.randint(case["steps_min"], case["steps_max"])
        eps = r.uniform(1e-3, 1e-2)
        data = None if seed is None else (nb.plummer if k % 2 else nb.hernquist)(n, seed=1000 * seed + k)
        got.append((n, steps, eps, data))
    return got


def _inputs(case, seed):
    if case["kind"] == "adaptive":
        return nb.collision(case["n_each"], seed=2 * seed)
    return _cluster(case, case["n"], seed)


def _probes(case, seed):
    return np.random.default_rng(2 * seed + 1).normal(0.0, 1.5, (case["points"], 3))


_ADAPTIVE = dict(TimeBegin=0.0, TimeEnd=40.0, TimeBase=1 << 30, ErrTolTimestep=0.025, MinStep=1e-12, MaxStep=1e-2)


def _simulation(case, data):
    kw = dict(ForceSofteningTable=[case["eps"]] * 6, precision=case.get("precision", "mixed"),
              law=case.get("law", "spline"))
    if case["kind"] == "adaptive":
        return nb.Simulation(data, criterion="eta_sqrt_eps", **_ADAPTIVE, **kw)
    return nb.Simulation(data, TimeStep=case.get("dt", 1e-3), TimeEnd=1e6, **kw)


def prepare(case, seed):
    if case["kind"] == "ensemble":
        s = _systems(case, seed)
        total = sum(n for n, _, _, _ in s)
        eng = nb.Engine(max_particles=total, max_systems=len(s), law=case["law"])
        return {"case": case, "engine": eng, "systems": s}
    sim = _simulation(case, _inputs(case, seed))
    st = {"case": case, "sim": sim, "out": torch.empty((10, sim.n), dtype=torch.float64, pin_memory=True)}
    if case["kind"] == "probe":
        st["points"] = _probes(case, seed)
    elif case["kind"] in ("step", "adaptive"):
        # the start of a run: first force, first bins, forward half kick
        nb.compute_force(sim)
        nb.init_timesteps(sim)
        nb.leapfrog_half_kick(sim, +1)
    return st


# ---- one pass -------------------------------------------------------------


def _download(st, rows):
    """Rows of (x, y, z, vx, vy, vz, ax, ay, az, pot) into the state's pinned buffer."""
    buf = st["out"]
    ptr = [ctypes.cast(buf[k].data_ptr(), ctypes.POINTER(ctypes.c_double)) if k in rows else None
           for k in range(10)]
    L.check(st["sim"].handle, L.load().nb_download(st["sim"].handle, *ptr, None, None))
    return buf


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        eng = state["engine"]
        ids = [eng.submit(d, eps, 1e-3, steps) for n, steps, eps, d in state["systems"]]
        eng.run_until_idle()
        got = [eng.fetch(i, s[0]) for i, s in zip(ids, state["systems"])]
        return {k: np.concatenate([g[k] for g in got]) for k in ("pos", "vel")}
    sim = state["sim"]
    if case["kind"] == "probe":
        acc, pot = nb.force_and_potential_at_points(sim, state["points"], case["eps"])
        return {"acc": acc.astype(np.float32), "pot": pot.astype(np.float32)}
    if case["kind"] == "snapshot":
        nb.compute_force(sim, want_potential=True)
        buf = _download(state, (6, 7, 8, 9))
        acc, pot = buf[6:9].float(), buf[9].float()
        e = nb.diagnostics(sim)
        return {"acc": acc, "pot": pot, "K": e["K"], "W": e["W"], "P": e["P"], "L": e["L"]}
    nb.step(sim, case["steps"])
    buf = _download(state, range(9))
    acc = buf[6:9] if case.get("precision") == "fp64" else buf[6:9].float()
    return {"pos": buf[0:3], "vel": buf[3:6], "acc": acc}


# ---- what a pass cannot do without ----------------------------------------


def work(case):
    # 20 operations for an interaction (differences, square, root, three sums), the direct sum's convention
    if case["kind"] == "ensemble":
        s = _systems(case)
        return {"bytes": 8.0 * 13 * sum(q[0] for q in s), "flops": 20.0 * sum(q[0] ** 2 * q[1] for q in s)}
    if case["kind"] == "probe":
        n, m = case["n"], case["points"]
        return {"bytes": 8.0 * (4 * n + 7 * m), "flops": 20.0 * n * m}
    if case["kind"] == "adaptive":
        # about a quarter of the particles are due at an average step
        n = 2 * case["n_each"]
        return {"bytes": 8.0 * 16 * n, "flops": 20.0 * n * n * case["steps"] / 4}
    n = case["n"]
    if case["kind"] == "snapshot":
        return {"bytes": 8.0 * (7 + 4) * n, "flops": 20.0 * 2 * n * n}
    return {"bytes": 8.0 * 16 * n, "flops": 20.0 * n * n * case["steps"]}


# ---- the same in 64 bits --------------------------------------------------


def _field64(tgt, pos, mass, h, law, want_pot=False):
    """Acceleration (and potential) of the sources at tgt, (3, M) and (3, N) FP64 tensors, G = 1."""
    acc, pot = torch.empty_like(tgt), torch.empty_like(tgt[0])
    rows = max(1, (1 << 27) // max(1, pos.shape[1]))
    for b in range(0, tgt.shape[1], rows):
        d = [pos[k][None, :] - tgt[k, b:b + rows][:, None] for k in range(3)]
        r2 = d[0] * d[0]
        r2 += d[1] * d[1]
        r2 += d[2] * d[2]
        if law == "plummer":
            inv = (r2 + h * h).rsqrt()
            w = mass * inv * inv * inv
            p = torch.where(r2 > 0, -mass * inv, torch.zeros_like(inv)) if want_pot else None
        else:
            inv = r2.clamp_min(1e-300).rsqrt()
            w = mass * inv * inv * inv
            p = -mass * inv if want_pot else None
            i, j = torch.nonzero(r2 < h * h, as_tuple=True)
            r, m = r2[i, j].sqrt(), mass[j]
            u = r / h
            s = u.clamp_min(0.5)
            outer = (21.333333333333 - 48 * s + 38.4 * s ** 2 - 10.666666666667 * s ** 3
                     - 0.066666666667 / s ** 3)
            w[i, j] = m / h ** 3 * torch.where(u < 0.5, 10.666666666667 + u * u * (32 * u - 38.4), outer)
            if want_pot:
                po = (-3.2 + 0.066666666667 / s
                      + s * s * (10.666666666667 + s * (-16 + s * (9.6 - 2.133333333333 * s))))
                pi = -2.8 + u * u * (5.333333333333 + u * u * (6.4 * u - 9.6))
                p[i, j] = torch.where(r > 0, m / h * torch.where(u < 0.5, pi, po), torch.zeros_like(r))
        for k in range(3):
            d[k] *= w
            acc[k, b:b + rows] = d[k].sum(1)
        if want_pot:
            pot[b:b + rows] = p.sum(1)
    return (acc, pot) if want_pot else acc


def _dev(a):
    return torch.tensor(np.ascontiguousarray(np.asarray(a).T), device="cuda")


def _kdk64(x, v, m, h, law, dt, steps):
    a = _field64(x, x, m, h, law)
    v = v + a * (0.5 * dt)
    for _ in range(steps):
        x = x + v * dt
        a = _field64(x, x, m, h, law)
        v = v + a * dt
    return x, v, a


def _adaptive64(x, v, m, h, steps):
    c = _ADAPTIVE
    base, unit = c["TimeBase"], (c["TimeEnd"] - c["TimeBegin"]) / c["TimeBase"]

    def bins(a):
        dt = (c["ErrTolTimestep"] * torch.sqrt(h / torch.sqrt((a * a).sum(0)))).clamp_max(c["MaxStep"])
        b = torch.full_like(dt, base, dtype=torch.int64)
        while bool((late := b.double() > dt / unit).any()):
            b = torch.where(late, b >> 1, b)
        return b

    a = _field64(x, x, m, h, "spline")
    beg, end, now = torch.zeros_like(x[0], dtype=torch.int64), bins(a), 0
    v = v + a * 0.5 * (end - beg).double() * unit
    for _ in range(steps):
        nxt = min(base, int(end.min()))
        x = x + v * ((nxt - now) * unit)
        now = nxt
        due = end == now
        a = a.clone()
        a[:, due] = _field64(x[:, due], x, m, h, "spline")
        ti = bins(a).clamp_max(base - now)
        dt = ((end.double() + 0.5 * ti.double()) - (beg + end).double() / 2) * unit
        v = torch.where(due, v + a * dt, v)
        beg, end = torch.where(due, end, beg), torch.where(due, end + ti, end)
    return x, v, a


def exact(case, seed):
    if case["kind"] == "ensemble":
        s = _systems(case, seed)
        if sum(max(q[0] ** 2, 4e6) * q[1] for q in s) > 1.5e11:
            return None
        pos, vel = [], []
        for n, steps, eps, d in s:
            x, v, a = _kdk64(_dev(d["pos"]), _dev(d["vel"]), _dev(d["mass"]), eps, case["law"], 1e-3, steps)
            pos.append(x.T.cpu())
            vel.append((v - a * 0.5e-3).T.cpu())
        return {"pos": torch.cat(pos), "vel": torch.cat(vel)}
    d = _inputs(case, seed)
    x, v, m, h = _dev(d["pos"]), _dev(d["vel"]), _dev(d["mass"]), case["eps"]
    if case["kind"] == "probe":
        acc, pot = _field64(_dev(_probes(case, seed)), x, m, h, case["law"], True)
        return {"acc": acc.T.cpu(), "pot": pot.cpu()}
    if case["kind"] == "adaptive":
        if (2.0 * case["n_each"]) ** 2 * case["steps"] > 6e10:
            return None
        x, v, a = _adaptive64(x, v, m, h, case["steps"])
    elif case["kind"] == "snapshot":
        if case["n"] > 250000:
            return None
        acc, pot = _field64(x, x, m, h, case["law"], True)
        c = torch.linalg.cross(x, v, dim=0)
        return {"acc": acc.cpu(), "pot": pot.cpu(), "K": float(0.5 * (m * (v * v).sum(0)).sum()),
                "W": float(0.5 * (m * pot).sum()), "P": (m * v).sum(1).cpu(), "L": (m * c).sum(1).cpu()}
    else:
        if float(case["n"]) ** 2 * (case["steps"] + 1) > 6e10:
            return None
        x, v, a = _kdk64(x, v, m, h, case["law"], case["dt"], case["steps"])
    return {"pos": x.cpu(), "vel": v.cpu(), "acc": a.cpu()}
