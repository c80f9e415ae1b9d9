"""The work a user of this engine has it do, as cases that can be timed.

Every case goes through the public entry points (the Python front end and the C
ABI under it).  A single simulation works in place on the caller's device
arrays (nb_bind_device), as the reference's calculators work on the caller's
ParticleArrays, so a pass's outputs are those arrays.  The mixed and the
Barnes-Hut methods compute accelerations in FP32 pair arithmetic and hold them
in FP64 planes; a pass hands them on as float32, the precision they carry.
Positions and velocities are FP64 throughout.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call
  run(state)          one pass
  work(case)          bytes and operations a pass cannot do without
  exact(case, seed)   what run returns, in 64-bit torch
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("n-body-gravity-simulation_gb300"))
import nbody_gb300 as nb  # noqa: E402

METHODS = {"fp64": nb.DIRECT_FP64, "mixed": nb.DIRECT_MIXED, "bh": nb.BARNES_HUT}
INTEGRATORS = {"euler_cromer": nb.EULER_CROMER, "leapfrog": nb.LEAPFROG,
               "verlet": nb.VELOCITY_VERLET, "rk4": nb.RK4}
FLAGS = {"": 0, "quadrupole": nb.BH_QUADRUPOLE, "reference_opening": nb.BH_REFERENCE_OPENING}
EVALS_PER_STEP = {"euler_cromer": 1, "leapfrog": 1, "verlet": 1, "rk4": 4}


def listed():
    return [
        # the smallest runs of the reference's test programs (its 100-body
        # particle file): a step is launches and latency
        _step("fp64_leapfrog_n100", "fp64", 100, "leapfrog", 0.01, 1e-3),
        # the CPU-runnable configuration: 1024-body Plummer sphere in FP64
        _step("fp64_leapfrog_n1024", "fp64", 1024, "leapfrog", 0.01, 1e-3, steps=10),
        # one FP64 force evaluation of host data (the reference's largest
        # particle file, 10,000 bodies): upload, forces, accelerations back
        dict(name="fp64_host_n10000", kind="host", n=10000, softening=0.01),
        # an ordinary small system on the mixed path
        _step("mixed_verlet_n1000", "mixed", 1000, "verlet", 1e-3, 5e-4),
        # a ragged mid-size system on the mixed path, four evaluations a step
        _step("mixed_rk4_n5003", "mixed", 5003, "rk4", 1e-3, 5e-4),
        # the mixed-precision configuration: 65,536-body Plummer sphere
        _step("mixed_verlet_n65536", "mixed", 65536, "verlet", 1e-3, 5e-4),
        # a large, ragged direct sum (checking a tree code's forces)
        dict(name="mixed_forces_n400003", kind="forces", method="mixed", n=400003,
             model="disk", softening=1e-3, theta=0.5, option=""),
        # the reference API's Barnes-Hut calculator (its opening rule) on an
        # ordinary disk galaxy
        _step("bh_reference_n100000", "bh", 100000, "leapfrog", 1e-3, 1e-3, model="disk",
              theta=0.5, option="reference_opening"),
        # the Barnes-Hut configuration: 2^20-body bulge + disk
        _step("bh_leapfrog_n1048576", "bh", 1 << 20, "leapfrog", 1e-3, 1e-3, model="disk",
              theta=0.5),
        # the batched-ensemble configuration on a quarter of its systems
        dict(name="ensemble_rk4_1024", kind="ensemble", systems=1024, lo=32, hi=4096,
             steps=2, softening=1e-3),
        # the serving configuration's job mix as one burst
        dict(name="serve_burst_16", kind="serve", jobs=16, lo=1024, hi=131072, steps=4),
        # the energy and momentum check between runs of steps
        dict(name="diagnostics_n20000", kind="diagnostics", n=20000, softening=1e-3),
    ]


def _step(name, method, n, integrator, softening, dt, steps=1, model="plummer", theta=0.5,
          option=""):
    c = dict(kind="step", method=method, n=n, integrator=integrator, softening=softening,
             dt=dt, steps=steps, model=model, theta=theta, option=option)
    if name:
        c["name"] = name
    return c


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    family = rng.choice(("fp64", "fp64_host", "mixed_small", "mixed_large", "mixed_forces",
                         "bh", "ensemble", "serve", "diagnostics"))
    eps = rng.choice((1e-3, 0.01))
    if family == "fp64":
        return _step(None, "fp64", _log_int(rng, 16, 8192),
                     rng.choice(("euler_cromer", "leapfrog", "verlet", "rk4")), eps, 1e-3,
                     steps=rng.choice((1, 4, 10)))
    if family == "fp64_host":
        return dict(kind="host", n=_log_int(rng, 100, 30000), softening=eps)
    if family == "mixed_small":
        return _step(None, "mixed", _log_int(rng, 100, 16383), rng.choice(("verlet", "rk4")),
                     eps, 5e-4, steps=rng.choice((1, 4)))
    if family == "mixed_large":
        return _step(None, "mixed", _log_int(rng, 16384, 150000),
                     rng.choice(("verlet", "leapfrog")), eps, 5e-4,
                     model=rng.choice(("plummer", "disk")))
    if family == "mixed_forces":
        return dict(kind="forces", method="mixed", n=_log_int(rng, 16384, 400000),
                    model=rng.choice(("plummer", "disk")), softening=eps, theta=0.5, option="")
    if family == "bh":
        return _step(None, "bh", _log_int(rng, 4096, 500000), "leapfrog", eps, 1e-3,
                     model=rng.choice(("plummer", "disk")), theta=rng.choice((0.5, 0.6, 0.8)),
                     option=rng.choice(("", "", "quadrupole", "reference_opening")))
    if family == "ensemble":
        return dict(kind="ensemble", systems=_log_int(rng, 24, 900), lo=32,
                    hi=rng.choice((1024, 4096)), steps=rng.choice((1, 2)), softening=eps)
    if family == "serve":
        return dict(kind="serve", jobs=rng.randint(3, 14), lo=1024,
                    hi=rng.choice((16384, 131072)), steps=rng.choice((2, 4)))
    return dict(kind="diagnostics", n=_log_int(rng, 64, 30000), softening=eps)


# ---------------------------------------------------------------- inputs
def _bodies(model, n, seed):
    """(x, y, z, vx, vy, vz, m), host float64."""
    return nb.plummer(n, seed=seed) if model == "plummer" else nb.disk_bulge(n, seed=seed)


def _job_sizes(case, seed):
    rng = np.random.default_rng(1000 + seed)
    u = (np.arange(case["jobs"]) + rng.uniform(size=case["jobs"])) / case["jobs"]
    return np.floor(case["lo"] * (case["hi"] / case["lo"]) ** u).astype(int)


def _sizes(case):
    # the sizes belong to the case, the bodies to the seed
    return nb.ensemble_sizes(case["systems"], case["lo"], case["hi"], 0)


def _bound(case, seed):
    """A simulation that works in place on ten rows of a device tensor."""
    n = case["n"]
    host = _bodies(case.get("model", "plummer"), n, seed)
    state = torch.zeros(10, -(-n // 32) * 32, dtype=torch.float64, device="cuda")
    for row, v in zip((0, 1, 2, 3, 4, 5, 9), host):
        state[row, :n] = torch.from_numpy(v)
    cfg = nb.Config(method=METHODS[case.get("method", "fp64")], G=1.0,
                    softening=case["softening"], theta=case.get("theta", 0.5),
                    flags=FLAGS[case.get("option", "")])
    sim = nb.Sim(cfg, capacity=n)
    rows = (nb.C.c_void_p * 10)(*[state[k].data_ptr() for k in range(10)])
    status = nb.lib().nb_bind_device(sim.handle, n, rows)
    if status != 0:
        raise nb.NBodyError(status, "nb_bind_device", "")
    return sim, state


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("step", "forces", "diagnostics"):
        s["sim"], s["state"] = _bound(case, seed)
    elif kind == "host":
        s["sim"] = nb.Sim(nb.Config(method=nb.DIRECT_FP64, G=1.0, softening=case["softening"]),
                          capacity=case["n"])
        s["host"] = [torch.from_numpy(v).pin_memory()
                     for v in _bodies("plummer", case["n"], seed)]
        s["acc"] = [torch.zeros(case["n"], dtype=torch.float64).pin_memory() for _ in range(3)]
    elif kind == "ensemble":
        sizes = _sizes(case)
        e = nb.Ensemble(nb.Config(method=nb.DIRECT_MIXED, G=1.0, softening=case["softening"]),
                        sizes)
        e.load(*nb.plummer_ensemble(sizes, seed=seed * 100003))
        s["ens"] = e
        s["out"] = torch.zeros(9, e.total, dtype=torch.float64).pin_memory()
    elif kind == "serve":
        s["jobs"] = [_bodies("plummer" if k % 2 == 0 else "disk", int(n), seed * 101 + k)
                     for k, n in enumerate(_job_sizes(case, 0))]
        s["server"] = nb.Server()
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        s["sim"].step(INTEGRATORS[case["integrator"]], case["dt"], case["steps"])
        return _state(case, s["state"])
    if kind == "forces":
        s["sim"].compute_forces()
        return s["state"][6:9, :case["n"]].float()
    if kind == "host":
        sim, n = s["sim"], case["n"]
        sim.load_pointers(n, [h.data_ptr() for h in s["host"]])
        sim.compute_forces()
        sim.read_pointers([0] * 6 + [a.data_ptr() for a in s["acc"]] + [0])
        return s["acc"]
    if kind == "ensemble":
        e, out = s["ens"], s["out"]
        e.step(nb.RK4, 1e-3, case["steps"])
        ptrs = [nb.C.c_void_p(out[k].data_ptr()) for k in range(6)]
        status = nb.lib().nb_ensemble_read_state(e._h, *ptrs, None, None, None, None)
        if status != 0:
            raise nb.NBodyError(status, "nb_ensemble_read_state", "")
        return out[:6]
    if kind == "serve":
        srv = s["server"]
        ids = [srv.submit(j, case["steps"]) for j in s["jobs"]]
        srv.run_until_idle()
        out = []
        for i in ids:
            r = srv.result(i)
            srv.release(i)
            out.append(np.stack([r[k] for k in ("x", "y", "z", "vx", "vy", "vz")]))
        return out
    d = s["sim"].diagnostics()
    return np.array([d["kinetic"], d["potential"], d["potential_softened"], d["total"],
                     d["total_softened"], d["mass"], *d["angular_momentum"],
                     *d["center_of_mass"], *d["momentum"]])


def _state(case, state):
    """Positions and velocities, and the accelerations (float32 where the
    method computes them in FP32 arithmetic; RK4 and Euler-Cromer leave the
    start-of-step ones)."""
    n = case["n"]
    acc = state[6:9, :n]
    return dict(state=state[:6, :n], acc=acc if case["method"] == "fp64" else acc.float())


# ---------------------------------------------------------------- work
FLOPS = 20.0  # per pair: displacement 3, r^2 6, r^-3 5, accumulation 6


def _terms_per_body(n, theta):
    return min(n - 1.0, 40.0 / theta ** 2 * math.log2(max(2.0, n / 8.0)))


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        sizes = _sizes(case).astype(float)
        evals = 4 * case["steps"]
        return dict(bytes=float(sizes.sum()) * (56 * case["steps"] * 2 + 48),
                    flops=FLOPS * evals * float((sizes * (sizes - 1)).sum()))
    if kind == "serve":
        flops = moved = 0.0
        for n in _job_sizes(case, 0).astype(float):
            terms = n - 1 if n < 16384 else _terms_per_body(n, 0.6)
            flops += FLOPS * n * terms * case["steps"]
            moved += n * (56 + 80 + 104 * case["steps"])
        return dict(bytes=moved, flops=flops)
    n = float(case["n"])
    if kind == "diagnostics":
        # half the pairs, two square roots and divisions each
        return dict(bytes=56 * n, flops=14.0 * n * (n - 1) / 2)
    if kind == "host":
        return dict(bytes=(56 + 24) * n, flops=FLOPS * n * (n - 1))
    terms = _terms_per_body(n, case["theta"]) if case["method"] == "bh" else n - 1
    if kind == "forces":
        return dict(bytes=(32 + 24) * n, flops=FLOPS * n * terms)
    evals = EVALS_PER_STEP[case["integrator"]] * case["steps"]
    return dict(bytes=(56 + 72) * n * case["steps"], flops=FLOPS * n * terms * evals)


# ---------------------------------------------------------------- 64-bit torch
def _exact_forces(p, m, eps2):
    """Accelerations (3, n) of positions p (3, n) by the direct sum."""
    n = p.shape[1]
    a = torch.empty_like(p)
    rows = max(1, min(n, (1 << 27) // n))
    for i in range(0, n, rows):
        d = p[:, None, :] - p[:, i:i + rows, None]
        r2 = (d * d).sum(0).add_(eps2)
        a[:, i:i + rows] = (d.mul_(m / (r2 * r2.sqrt()))).sum(-1)
    return a


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve" or (kind != "ensemble" and case["n"] > 420000):
        return None  # a tree code's own approximation; too many pairs
    if kind == "ensemble":
        if case["systems"] > 1100:
            return None
        sizes = _sizes(case)
        rows = torch.from_numpy(np.stack(nb.plummer_ensemble(sizes, seed=seed * 100003))).cuda()
        out, at = [], 0
        for n in sizes:
            part = rows[:, at:at + int(n)]
            p, v, _ = _exact_steps(part[:3], part[3:6], part[6], "rk4", 1e-3, case["steps"],
                                   case["softening"] ** 2)
            out.append(torch.cat([p, v]))
            at += int(n)
        return torch.cat(out, 1)
    host = torch.from_numpy(np.stack(_bodies(case.get("model", "plummer"), case["n"],
                                             seed))).cuda()
    p, v, m = host[:3], host[3:6], host[6]
    eps2 = case["softening"] ** 2
    if kind == "forces":
        return _exact_forces(p, m, eps2)
    if kind == "host":
        return list(_exact_forces(p, m, eps2))
    if kind == "diagnostics":
        return _exact_diagnostics(p, v, m, eps2)
    if case["method"] == "bh":
        # the tree's own error is in the accelerations; over one short step
        # positions and velocities are held to their type alone
        return dict(state=None, acc=_exact_steps(p, v, m, case["integrator"], case["dt"],
                                                 case["steps"], eps2)[2])
    p, v, a = _exact_steps(p, v, m, case["integrator"], case["dt"], case["steps"], eps2)
    return dict(state=torch.cat([p, v]), acc=a)


def _exact_steps(p, v, m, integrator, dt, steps, eps2):
    a = None
    for _ in range(steps):
        if integrator == "euler_cromer":
            a = _exact_forces(p, m, eps2)
            v = v + a * dt
            p = p + v * dt
        elif integrator == "leapfrog":
            a = _exact_forces(p, m, eps2) if a is None else a
            v = v + a * (dt / 2)
            p = p + v * dt
            a = _exact_forces(p, m, eps2)
            v = v + a * (dt / 2)
        elif integrator == "verlet":
            old = _exact_forces(p, m, eps2) if a is None else a
            p = p + (v * dt + old * 0.5 * dt * dt)
            a = _exact_forces(p, m, eps2)
            v = v + (old + a) * (0.5 * dt)
        else:
            h = dt / 2
            a = _exact_forces(p, m, eps2)
            v2 = v + a * h
            a2 = _exact_forces(p + v * h, m, eps2)
            v3 = v + a2 * h
            a3 = _exact_forces(p + v2 * h, m, eps2)
            v4 = v + a3 * dt
            a4 = _exact_forces(p + v3 * dt, m, eps2)
            p = p + (v + 2 * v2 + 2 * v3 + v4) * (dt / 6)
            v = v + (a + 2 * a2 + 2 * a3 + a4) * (dt / 6)
    return p, v, a


def _exact_diagnostics(p, v, m, eps2):
    n = p.shape[1]
    pu, ps = torch.zeros_like(m), torch.zeros_like(m)
    rows = max(1, min(n, (1 << 26) // n))
    for i in range(0, n, rows):
        d = p[:, None, :] - p[:, i:i + rows, None]
        r2 = (d * d).sum(0)
        k = torch.arange(r2.shape[0], device=r2.device)
        u = m / r2.sqrt()
        u[k, k + i] = 0.0
        w = m / (r2 + eps2).sqrt()
        w[k, k + i] = 0.0
        pu[i:i + rows], ps[i:i + rows] = u.sum(-1), w.sum(-1)
    kin = float((0.5 * m * (v * v).sum(0)).sum())
    pot, soft = -0.5 * float((m * pu).sum()), -0.5 * float((m * ps).sum())
    mass = float(m.sum())
    ang = torch.linalg.cross(p, v, dim=0) * m
    com, mom = (p * m).sum(1) / mass, (v * m).sum(1)
    return np.array([kin, pot, soft, kin + pot, kin + soft, mass, *ang.sum(1).tolist(),
                     *com.tolist(), *mom.tolist()])
