"""Workloads that stand for what this library is used for.

``listed()`` names them, ``draw()`` gives more of the same ranges,
``prepare()`` makes what a program holds before the call, ``run()`` is one
pass through the public entry points, ``work()`` what a pass cannot do
without, and ``exact()`` the same quantities by all-pairs summation in 64 bits
(the value the tree approximates), written in plain torch.

Sizes and parameters are those of the repository's own workloads (bench.py,
nbb/workloads.py, the tests): Plummer spheres, disk + bulge, Gaussian blobs
and ensembles, theta 0.3 .. 0.7, 10^3 .. 2^22 particles.

The mixed form evaluates forces in FP32, so a program that uses it takes the
accelerations, velocity updates and gradients it gets in FP32; ``run()``
returns them so.  Its warp group size is part of a case: the default lets the
library time 32, 64 and 128 and keep the fastest, which makes the interaction
lists depend on a timing.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "amsc-nbody_b200"))

import nbb  # noqa: E402
from nbb import ics  # noqa: E402

DT = 1e-3
FIELDS = ("mass", "x", "y", "z", "vx", "vy", "vz")


def listed():
    return [
        # interactive and test-sized systems: latency and launches decide
        dict(name="step_fp64_1000", kind="run", shape="plummer", n=1000, theta=0.5, eps=0.01, mixed=False, steps=1),
        dict(name="run_mixed_4096", kind="run", shape="plummer", n=4096, theta=0.5, eps=0.01, mixed=True, group=32, steps=8),
        # a cluster advanced a few steps between snapshots
        dict(name="run_mixed_65536", kind="run", shape="plummer", n=65536, theta=0.5, eps=0.01, mixed=True, group=32, steps=4),
        # the benchmark's system in both forms, one step at a time
        dict(name="step_mixed_1048576", kind="run", shape="plummer", n=1048576, theta=0.5, eps=0.01, mixed=True, group=64, steps=1),
        dict(name="step_fp64_1048576", kind="run", shape="plummer", n=1048576, theta=0.5, eps=0.01, mixed=False, steps=1),
        # a galaxy: flat, dense in the middle, an odd particle count
        dict(name="step_fp64_disk_300007", kind="run", shape="disk", n=300007, theta=0.7, eps=0.005, mixed=False, steps=1),
        # the largest system: clustered, unequal masses, cold start
        dict(name="step_mixed_blobs_4194304", kind="run", shape="blobs", n=4194304, theta=0.5, eps=1e-3, mixed=True, group=64, steps=1),
        # many independent systems of very different sizes in one handle
        dict(name="ensemble_mixed_64", kind="ensemble", systems=64, n_min=1024, n_max=131072, theta=0.5, mixed=True, group=32, steps=1),
        # one force evaluation of host arrays (analysis scripts, other integrators)
        dict(name="force_fp64_host_50021", kind="force", shape="plummer", n=50021, theta=0.5, eps=0.01, mixed=False),
        # a host program that owns the state between steps
        dict(name="host_step_mixed_262144", kind="host_step", shape="plummer", n=262144, theta=0.5, eps=0.01, mixed=True, group=64),
        # rollouts and their gradients (fitting initial conditions)
        dict(name="gradient_mixed_65536", kind="gradient", shape="plummer", n=65536, theta=0.5, eps=0.01, mixed=True, group=32, steps=8, every=4),
        dict(name="gradient_fp64_16384", kind="gradient", shape="plummer", n=16384, theta=0.5, eps=0.01, mixed=False, steps=8, every=4),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 5 + ["ensemble", "force", "host_step", "gradient"])
    theta = rng.choice([0.3, 0.5, 0.5, 0.5, 0.7])
    mixed = rng.random() < 0.5
    if kind == "ensemble":
        return dict(kind=kind, systems=rng.randint(2, 96), n_min=1024, n_max=_log_uniform(rng, 2048, 65536),
                    theta=0.5, mixed=mixed, group=32, steps=1)
    top = {"run": 3000000 if mixed else 1048576, "force": 262144, "host_step": 1048576, "gradient": 65536}[kind]
    n = _log_uniform(rng, 1000, top)
    shape = rng.choice(["plummer", "plummer", "disk", "blobs"])
    if kind in ("host_step", "gradient") or (shape == "blobs" and not mixed and n > 400000):
        shape = "plummer"
    if n > 400000:
        theta = max(theta, 0.5)
    case = dict(kind=kind, shape=shape, n=n, theta=theta, eps={"plummer": 0.01, "disk": 0.005, "blobs": 1e-3}[shape],
                mixed=mixed)
    if mixed and kind != "force":
        # what the library's own tuning picks at these sizes
        case["group"] = 32 if n < 131072 else rng.choice([64, 128])
    if kind == "run":
        case["steps"] = rng.randint(1, 8) if n < 131072 else 1
    if kind == "gradient":
        case["steps"] = rng.randint(2, 8)
        case["every"] = rng.randint(1, 4)
    return case


# ---------------------------------------------------------------- inputs ---

def _particles(case, seed):
    if case["kind"] == "ensemble":
        sizes = _sizes(case)
        parts = [ics.plummer(int(k), seed=seed * 1009 + s) for s, k in enumerate(sizes)]
        return ics.ParticleData(*(np.concatenate([getattr(p, f) for p in parts]) for f in FIELDS))
    make = {"plummer": ics.plummer, "disk": ics.disk_bulge, "blobs": ics.blobs}[case["shape"]]
    return make(case["n"], seed=seed)


def _sizes(case):
    """System sizes log-uniform in [n_min, n_max], in a fixed scattered order."""
    k = case["systems"]
    u = (np.arange(k) * 0.6180339887498949) % 1.0
    return np.rint(case["n_min"] * (case["n_max"] / case["n_min"]) ** u).astype(np.int64)


def _ensemble_eps(case):
    return 0.01 * (4096.0 / _sizes(case)) ** (1.0 / 3.0)


def _config(case):
    return nbb.SimulationConfig(DT, case["theta"], case.get("eps", 0.0), 1.0,
                                precision=nbb.PRECISION_MIXED if case["mixed"] else nbb.PRECISION_FP64,
                                group_size=case.get("group", 0))


class _DeviceArray:
    """A device pointer of a simulation as torch.as_tensor takes it; the
    tensor keeps this object, and so the simulation that owns the memory."""

    def __init__(self, sim, pointer, n):
        self.sim = sim
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(pointer, False), version=2)


def _views(sim, n):
    v = sim.particles()
    return {f: torch.as_tensor(_DeviceArray(sim, getattr(v, f), n), device="cuda")
            for f in ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")}


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _cotangents(case, seed):
    """dL/d(final positions) and dL/d(final velocities) of a mean-square loss
    against a target some distance away."""
    rng = np.random.Generator(np.random.Philox(seed + 777))
    return rng.standard_normal((3, case["n"])) / case["n"], rng.standard_normal((3, case["n"])) / case["n"]


def prepare(case, seed):
    p = _particles(case, seed)
    kind = case["kind"]
    state = {"case": case, "particles": p}
    if kind == "force":
        return state
    if kind == "ensemble":
        offsets = np.concatenate([[0], np.cumsum(_sizes(case))]).astype(np.int64)
        sim = nbb.EnsembleSimulation(ics.Ensemble(p, offsets, _ensemble_eps(case)), _config(case))
    else:
        sim = nbb.Simulation(p, _config(case))
    sim.initialize()
    state["sim"] = sim
    if kind in ("run", "ensemble"):
        state["views"] = _views(sim, len(p))
    elif kind == "host_step":
        state["host"] = [_pinned(a) for a in p.arrays()]
    elif kind == "gradient":
        state["cotangents"] = _cotangents(case, seed)
    return state


# ------------------------------------------------------------------ pass ---

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "force":
        a = nbb.compute_accelerations(state["particles"], case["theta"], case["eps"], 1.0,
                                      precision=nbb.PRECISION_MIXED if case["mixed"] else nbb.PRECISION_FP64)
        return [v.astype(np.float32) for v in a] if case["mixed"] else list(a)
    sim = state["sim"]
    if kind in ("run", "ensemble"):
        sim.run(case["steps"])
        views = state["views"]
        if not case["mixed"]:
            return views
        return {f: t if f in ("x", "y", "z") else t.float() for f, t in views.items()}
    if kind == "host_step":
        host = state["host"]
        return sim.step_host(mass=host[0], x=host[1], y=host[2], z=host[3], vx=host[4], vy=host[5], vz=host[6],
                             out=host[1:])
    # a rollout from the current state, then the gradient of a loss of its end
    gp, gv = state["cotangents"]
    sim.rollout(case["steps"], case["every"])
    gm, gx, gvel = sim.backward(gp, gv)
    out = {"mass": gm, "positions": gx, "velocities": gvel}
    return {k: v.astype(np.float32) for k, v in out.items()} if case["mixed"] else out


# ------------------------------------------------------------------ work ---

def _interactions(n, theta):
    """Interactions per target a Barnes-Hut walk of this opening angle needs,
    about (the plain form's count at 2^20 particles and theta 0.5 is 2100)."""
    return min(float(n), 105.0 * math.log2(max(n, 2)) * (0.5 / theta) ** 2)


def work(case):
    """Bytes: the state once in and once out.  Flops: 20 per interaction (the
    usual count of a softened point-mass term); a reverse step evaluates the
    force and its vector-Jacobian product (35 per interaction) once more."""
    steps = case.get("steps", 1)
    if case["kind"] == "ensemble":
        sizes = [int(k) for k in _sizes(case)]
        n = sum(sizes)
        pairs = sum(k * _interactions(k, case["theta"]) for k in sizes)
    else:
        n = case["n"]
        pairs = n * _interactions(n, case["theta"])
    if case["kind"] == "force":
        return {"bytes": 56.0 * n, "flops": 20.0 * pairs}
    if case["kind"] == "gradient":
        return {"bytes": (152.0 + 56.0 + 48.0) * n * steps, "flops": (20.0 + 20.0 + 35.0) * pairs * steps}
    return {"bytes": 152.0 * n * steps, "flops": 20.0 * pairs * steps}


# ----------------------------------------------------------------- exact ---

_CHUNK = 1 << 25  # pairs at a time


def _direct(m, x, eps):
    """All-pairs accelerations of positions x (3, n), FP64."""
    n = x.shape[1]
    a = torch.empty_like(x)
    rows = max(1, _CHUNK // n)
    for i in range(0, n, rows):
        d = x[:, None, :] - x[:, i:i + rows, None]
        r2 = (d * d).sum(0) + eps * eps
        f = m / (r2 * r2.sqrt())
        a[:, i:i + rows] = (d * torch.where(r2 > 0, f, torch.zeros_like(f))).sum(2)
    return a


def _direct_vjp(m, x, eps, c):
    """Gradient of sum(c * _direct(m, x)) with respect to m and x."""
    n = x.shape[1]
    gm, gx = torch.zeros_like(m), torch.zeros_like(x)
    rows = max(1, _CHUNK // n)
    for i in range(0, n, rows):
        d = x[:, None, :] - x[:, i:i + rows, None]
        ci = c[:, i:i + rows, None]
        r2 = (d * d).sum(0) + eps * eps
        inv3 = 1.0 / (r2 * r2.sqrt())
        dot = (d * ci).sum(0)
        gm += (inv3 * dot).sum(0)
        u = m * inv3 * (ci - 3.0 * (dot / r2) * d)
        gx += u.sum(1)
        gx[:, i:i + rows] -= u.sum(2)
    return gm, gx


def _leapfrog(m, x, v, eps, steps):
    """Kick-drift-kick; positions of every step, final velocities and
    accelerations."""
    xs, a = [x], _direct(m, x, eps)
    for _ in range(steps):
        v = v + 0.5 * DT * a
        x = x + DT * v
        a = _direct(m, x, eps)
        v = v + 0.5 * DT * a
        xs.append(x)
    return xs, v, a


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble" or case["n"] > (131072 if kind != "gradient" else 65536):
        return None
    if case["n"] ** 2 * (case.get("steps", 1) + 1) * (4 if kind == "gradient" else 1) > 1.6e11:
        return None
    p = _particles(case, seed)
    m = torch.from_numpy(p.mass).cuda()
    x = torch.from_numpy(np.stack([p.x, p.y, p.z])).cuda()
    v = torch.from_numpy(np.stack([p.vx, p.vy, p.vz])).cuda()
    eps = case["eps"]
    if kind == "force":
        return [a.cpu().numpy() for a in _direct(m, x, eps)]
    xs, v, a = _leapfrog(m, x, v, eps, case.get("steps", 1))
    if kind == "run":
        return dict(zip(("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az"), [*xs[-1], *v, *a]))
    if kind == "host_step":
        return [t.cpu().numpy() for t in (*xs[-1], *v)]
    gx, gv = (torch.from_numpy(c).cuda() for c in _cotangents(case, seed))
    gm = torch.zeros_like(m)
    for s in range(case["steps"], -1, -1):
        # closing kick of step s and opening kick of step s + 1 share a(x_s)
        w = 0.5 * DT if s in (0, case["steps"]) else DT
        dm, dx = _direct_vjp(m, xs[s], eps, w * gv)
        gm, gx = gm + dm, gx + dx
        if s:
            gv = gv + DT * gx
    return {"mass": gm.cpu().numpy(), "positions": gx.cpu().numpy(), "velocities": gv.cpu().numpy()}
