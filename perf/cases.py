"""Performance cases of the force-and-step path.

A case is one pass of work that a user of the library has it do: a force
evaluation or a leapfrog step on device arrays, a few steps of a simulation
handle with the new state read back, a batch of encounters advanced together,
an energy diagnostic.  ``listed()`` gives the fixed cases, ``draw()`` more of
the same ranges; ``prepare()`` makes what a program holds before the call,
``run()`` is one pass, ``exact()`` the same outputs from plain FP64 torch.
"""
import ctypes
import math

import numpy as np
import torch

from nbodyssey_b200 import _lib as L
from nbodyssey_b200 import api, ensemble, ic

DT = 0.005

# ---------------------------------------------------------------------------
# The cases.
#
# kind "forces": nb_compute_forces_dev, a(x) on caller-owned device arrays.
# kind "step":   nb_leapfrog_step_dev, one kick-drift-kick from a held state.
# kind "sim":    Simulation.step(steps), then the new positions and velocities
#                read back, the cadence of a run that writes frames.
# kind "batch":  Ensemble.step(steps) of independent encounters, states read.
# kind "energy": nb_total_energy_dev, the diagnostic of the energy log.
# ---------------------------------------------------------------------------


def _forces(name, n, force, traverse="warp", theta=0.5, key_bits=30, cores=False):
    return {"name": name, "kind": "forces", "n": n, "force": force, "traverse": traverse,
            "theta": theta, "key_bits": key_bits, "cores": cores}


def listed():
    return [
        # a call per step from a host that integrates a small system itself:
        # launches and latency are all of it
        _forces("naive_1k", 1000, "naive"),
        # the plain all-pairs workload, N = 12,000, run with frames: ten steps
        # through the handle's step graph, then the state comes back
        {"name": "naive_12k_steps", "kind": "sim", "n": 12000, "force": "naive",
         "traverse": "thread", "theta": 0.5, "steps": 10},
        # an all-pairs sweep point, odd size: neither a tile nor a warp multiple
        _forces("naive_50k_odd", 50001, "naive"),
        # the exact forces the precision study compares with, at its full size
        _forces("naive_262k", 262144, "naive", cores=True),
        # Barnes-Hut just above the all-pairs crossover, ragged
        _forces("bh_warp_20k_odd", 20011, "bh"),
        # the 100,000-particle Barnes-Hut run with frames
        {"name": "bh_warp_100k_steps", "kind": "sim", "n": 100000, "force": "bh",
         "traverse": "warp", "theta": 0.5, "steps": 10},
        # the wide-angle point of the theta sweep, thread semantics (the default)
        _forces("bh_thread_100k_t08", 100000, "bh", traverse="thread", theta=0.8),
        # the precision study's Barnes-Hut side: dense cores, full-width keys,
        # the theta that meets its energy gate
        _forces("bh_warp_262k_k63_t035", 262144, "bh", theta=0.35, key_bits=63, cores=True),
        # thread semantics at a sweep point, odd size
        _forces("bh_thread_400k_odd", 400003, "bh", traverse="thread"),
        # the headline workload: one leapfrog step of 1,000,000 particles
        {"name": "bh_warp_1m_step", "kind": "step", "n": 1000000, "force": "bh",
         "traverse": "warp", "theta": 0.5, "key_bits": 30},
        # an ensemble of encounters of many sizes, force module chosen by size
        {"name": "batch_24_steps", "kind": "batch", "sims": 24, "n_hi": 65536, "mix": 1,
         "steps": 20},
        # one row of the energy log of the 100,000-particle run
        {"name": "energy_100k", "kind": "energy", "n": 100000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: sizes log-uniform and mostly odd."""
    kind = rng.choice(["forces_naive", "forces_bh", "forces_bh", "forces_bh", "step", "sim",
                       "batch", "energy"])
    if kind == "forces_naive":
        return {"kind": "forces", "n": _log_uniform(rng, 256, 200000), "force": "naive",
                "traverse": "warp", "theta": 0.5, "key_bits": 30,
                "cores": rng.random() < 0.25}
    if kind == "forces_bh":
        return {"kind": "forces", "n": _log_uniform(rng, 4096, 1000000), "force": "bh",
                "traverse": rng.choice(["warp", "thread"]),
                "theta": rng.choice([0.35, 0.5, 0.5, 0.7, 0.8]),
                "key_bits": rng.choice([30, 30, 63]), "cores": rng.random() < 0.25}
    if kind == "step":
        return {"kind": "step", "n": _log_uniform(rng, 20000, 1000000), "force": "bh",
                "traverse": rng.choice(["warp", "thread"]), "theta": rng.choice([0.5, 0.7]),
                "key_bits": rng.choice([30, 30, 63])}
    if kind == "sim":
        n = _log_uniform(rng, 1000, 200000)
        return {"kind": "sim", "n": n, "force": "naive" if n < 16000 else "bh",
                "traverse": rng.choice(["warp", "thread"]), "theta": 0.5,
                "steps": rng.choice([5, 10])}
    if kind == "batch":
        return {"kind": "batch", "sims": rng.randint(6, 28),
                "n_hi": rng.choice([16384, 32768, 65536]), "mix": rng.randrange(1000),
                "steps": rng.choice([10, 20])}
    return {"kind": "energy", "n": _log_uniform(rng, 20000, 262144)}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
_started = False


def _start():
    """What a program does once: a first simulation, which loads the kernels
    and the tuning table that every later call on the device uses."""
    global _started
    if not _started:
        pos, vel = ic.two_disks(64, seed=0)
        api.Simulation(pos, vel, api.SimParams(force="naive")).close()
        _started = True


def _eps(case):
    return 0.01 if case.get("cores") else 0.05


def _state(case, seed):
    if case.get("cores"):
        return ic.precision_config(case["n"], seed=seed)
    return ic.two_disks(case["n"], seed=seed)


def _held_acc(pos):
    """The acceleration a held state comes with: each galaxy as one softened
    point mass (a program hands in the a(x) of its last step)."""
    p = torch.from_numpy(pos).double()
    a = torch.zeros_like(p)
    for cx, cy in ((-10.0, -2.0), (10.0, 2.0)):
        d = torch.tensor([cx, cy, 0.0], dtype=torch.float64) - p[:, :3]
        a[:, :3] += d / (d.square().sum(1, keepdim=True) + 1.0).pow(1.5)
    return a.float()


def _specs(case, seed):
    """The encounters of a batch: sizes from the case, the rest from the seed."""
    sizes = ic.ensemble_specs(case["sims"], seed=case["mix"], n_lo=2048, n_hi=case["n_hi"])
    specs = ic.ensemble_specs(case["sims"], seed=seed)
    return [dict(s, n=z["n"]) for s, z in zip(specs, sizes)]


def _params(case):
    return api.SimParams(dt=DT, epsilon=_eps(case), theta=case.get("theta", 0.5),
                         force=case.get("force", "naive"),
                         traverse=case.get("traverse", "warp"),
                         key_bits=case.get("key_bits", 30))


class _Workspace:
    """A device-pointer caller's scratch, kept with its arrays."""

    def __init__(self):
        self.lib = L.load()
        self.h = ctypes.c_void_p()
        L.check(self.lib.nb_workspace_create(ctypes.byref(self.h)))

    def __del__(self):
        self.lib.nb_workspace_destroy(self.h)


def prepare(case, seed):
    _start()
    kind = case["kind"]
    if kind == "batch":
        specs = _specs(case, seed)
        states = [ic.from_spec(s) for s in specs]
        params = [api.SimParams(dt=DT, epsilon=0.05, theta=0.5, force="auto",
                                traverse="warp" if i % 4 else "thread")
                  for i in range(len(specs))]
        return {"kind": kind, "ens": ensemble.Ensemble(states, params), "steps": case["steps"]}
    pos, vel = _state(case, seed)
    if kind == "sim":
        return {"kind": kind, "sim": api.Simulation(pos, vel, _params(case)),
                "steps": case["steps"]}
    dev = torch.device("cuda")
    s = {"kind": kind, "n": case["n"], "ws": _Workspace(), "p": _params(case).to_c(),
         "pos": torch.from_numpy(pos).to(dev)}
    if kind == "forces":
        s["acc"] = torch.zeros_like(s["pos"])
    else:
        s["vel"] = torch.from_numpy(vel).to(dev)
    if kind == "step":
        s["acc"] = _held_acc(pos).to(dev)
        s["out"] = [torch.empty_like(s["pos"]) for _ in range(3)]
    return s


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    kind = s["kind"]
    if kind == "batch":
        e = s["ens"]
        e.step(s["steps"])
        states = [e.state(i) for i in range(e.nsims)]
        return {"pos": np.concatenate([p for p, _ in states]),
                "vel": np.concatenate([v for _, v in states])}
    if kind == "sim":
        s["sim"].step(s["steps"])
        return {"pos": s["sim"].positions(), "vel": s["sim"].velocities()}
    lib = s["ws"].lib
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "forces":
        L.check(lib.nb_compute_forces_dev(s["ws"].h, s["n"], _ptr(s["pos"]), _ptr(s["acc"]),
                                          ctypes.byref(s["p"]), st))
        return s["acc"]
    if kind == "step":
        pos, vel, acc = s["out"]
        pos.copy_(s["pos"])
        vel.copy_(s["vel"])
        acc.copy_(s["acc"])
        L.check(lib.nb_leapfrog_step_dev(s["ws"].h, s["n"], _ptr(pos), _ptr(vel), _ptr(acc),
                                         ctypes.byref(s["p"]), st))
        return {"pos": pos, "vel": vel, "acc": acc}
    e3 = np.zeros(3, np.float64)
    L.check(lib.nb_total_energy_dev(s["ws"].h, s["n"], _ptr(s["pos"]), _ptr(s["vel"]),
                                    ctypes.byref(s["p"]), L.ptr(e3), st))
    return e3


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------
def _force_flops(n, force, traverse, theta):
    """20 flop per pair.  Barnes-Hut pairs per target: a fit, within a few per
    cent, of the counts the opening test gives on the two-disk state from
    4,096 to 1,000,000 particles at theta 0.3 to 0.8; a warp's shared set is
    about 1.7 times as long."""
    if force == "naive":
        return 20.0 * n * n
    lg = math.log2(max(n, 512) / 256.0)
    pairs = min(float(n), (24.0 + 2.5 * lg) * lg * (0.5 / theta) ** 2.2)
    return 20.0 * n * min(float(n), pairs * (1.7 if traverse == "warp" else 1.0))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        steps, flops, total = case["steps"], 0.0, 0
        for s in _specs(case, 1):
            flops += min(_force_flops(s["n"], "naive", "", 0.5),
                         _force_flops(s["n"], "bh", "warp", 0.5))
            total += s["n"]
        return {"bytes": 2.0 * 32.0 * total, "flops": steps * flops}
    n = case["n"]
    if kind == "energy":
        return {"bytes": 32.0 * n, "flops": 0.5 * 10.0 * n * n}
    f = _force_flops(n, case["force"], case["traverse"], case["theta"])
    if kind == "forces":
        return {"bytes": 32.0 * n, "flops": f}
    if kind == "step":
        return {"bytes": 96.0 * n, "flops": f}
    return {"bytes": 64.0 * n, "flops": case["steps"] * f}


# ---------------------------------------------------------------------------
# The outputs in FP64: direct sums over all pairs.  Barnes-Hut outputs are
# held to them too; their distance is the opening angle's.
# ---------------------------------------------------------------------------
_PAIRS_MAX = 1.3e11   # well under 20 seconds of pairs


def _acc64(x, m, eps2):
    """a_i = sum_j m_j (x_j - x_i) (r_ij^2 + eps2)^-1.5, rows in chunks."""
    n = x.shape[0]
    out = torch.empty_like(x)
    sq = x.square().sum(1)
    src = torch.cat([x * m[:, None], m[:, None]], 1)
    for i in range(0, n, rows := max(1, min(n, (1 << 27) // n))):
        xi = x[i:i + rows]
        r2 = torch.addmm(sq[None, :] + eps2, xi, x.t(), alpha=-2.0)
        r2.add_(sq[i:i + rows, None]).clamp_(min=eps2)
        w = r2.rsqrt_()
        s = torch.mm(w.square().mul_(w), src)
        out[i:i + rows] = s[:, :3] - xi * s[:, 3:]
    return out


def _phi64(x, m, eps2):
    n = x.shape[0]
    phi = torch.empty(n, dtype=torch.float64, device=x.device)
    sq = x.square().sum(1)
    for i in range(0, n, rows := max(1, min(n, (1 << 27) // n))):
        xi = x[i:i + rows]
        r2 = torch.addmm(sq[None, :] + eps2, xi, x.t(), alpha=-2.0)
        r2.add_(sq[i:i + rows, None]).clamp_(min=eps2)
        w = r2.rsqrt_()
        w[torch.arange(xi.shape[0]), torch.arange(i, i + xi.shape[0])] = 0.0
        phi[i:i + rows] = w @ m
    return phi


def _steps64(pos, vel, eps2, steps):
    dev = torch.device("cuda")
    x = torch.from_numpy(pos[:, :3]).double().to(dev)
    m = torch.from_numpy(pos[:, 3]).double().to(dev)
    v = torch.from_numpy(vel[:, :3]).double().to(dev)
    dt = float(np.float32(DT))
    a = _acc64(x, m, eps2)
    for _ in range(steps):
        v = v + 0.5 * dt * a
        x = x + dt * v
        a = _acc64(x, m, eps2)
        v = v + 0.5 * dt * a
    w = torch.from_numpy(vel[:, 3:]).double().to(dev)
    return torch.cat([x, m[:, None]], 1), torch.cat([v, w], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        specs = _specs(case, seed)
        if sum(s["n"] ** 2 for s in specs) * (case["steps"] + 1) > _PAIRS_MAX:
            return None
        got = [_steps64(*ic.from_spec(s), float(np.float32(0.05)) ** 2, case["steps"])
               for s in specs]
        return {"pos": torch.cat([p for p, _ in got]), "vel": torch.cat([v for _, v in got])}
    n = case["n"]
    if float(n) * n * (case.get("steps", 0) + 1) > _PAIRS_MAX:
        return None
    pos, vel = _state(case, seed)
    eps2 = float(np.float32(_eps(case))) ** 2
    if kind == "sim":
        p, v = _steps64(pos, vel, eps2, case["steps"])
        return {"pos": p, "vel": v}
    dev = torch.device("cuda")
    x = torch.from_numpy(pos[:, :3]).double().to(dev)
    m = torch.from_numpy(pos[:, 3]).double().to(dev)
    if kind == "forces":
        return torch.cat([_acc64(x, m, eps2), torch.zeros_like(m)[:, None]], 1)
    v = torch.from_numpy(vel[:, :3]).double().to(dev)
    if kind == "energy":
        ke = 0.5 * (m * v.square().sum(1)).sum()
        pe = -0.5 * (m * _phi64(x, m, eps2)).sum()
        return torch.stack([ke + pe, ke, pe])
    a = _held_acc(pos)[:, :3].double().to(dev)
    dt = float(np.float32(DT))
    v = v + 0.5 * dt * a
    x = x + dt * v
    a = _acc64(x, m, eps2)
    v = v + 0.5 * dt * a
    w = torch.from_numpy(vel[:, 3:]).double().to(dev)
    return {"pos": torch.cat([x, m[:, None]], 1), "vel": torch.cat([v, w], 1),
            "acc": torch.cat([a, torch.zeros_like(m)[:, None]], 1)}
