"""The all-pairs kernels: a warp per few targets below n = 2,560 (2 or 4
targets a warp by size, 8 in a batch; sources in batches of 128), each unordered pair once
from there on: tile and chunk edges, masses equal and not, ranges of scale, and
passes over a scratch too small for the whole table of partials."""
import numpy as np
import pytest

from nbodyssey_b200 import api, ic
from nbodyssey_b200.ensemble import Ensemble
from nbodyssey_b200.server import Server
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EPS = 0.05


def _rel(acc, exact):
    return np.linalg.norm(acc - exact, axis=1) / np.linalg.norm(exact, axis=1)


def _forces(pos, eps=EPS):
    prm = api.SimParams(epsilon=eps, force="naive")
    with api.Simulation(pos, np.zeros_like(pos), prm) as sim:
        return sim.compute_forces()


# the small kernel's batches and target counts, then both sides of every tile
# size and ragged last tiles and chunks
@pytest.mark.parametrize("n", [127, 128, 129, 1184, 1185, 2047, 2048, 2049, 2304, 2305, 2559, 2560, 2561,
                               4097, 8191, 8192, 8193, 8448, 8449, 16384, 16385, 24576, 24577,
                               65536, 65537, 163840, 163841])
@pytest.mark.parametrize("masses", ["equal", "spread"])
def test_sizes_vs_fp64(n, masses):
    pos, _ = ic.two_disks(n, seed=n)
    if masses == "spread":
        rng = np.random.default_rng(n)
        pos[:, 3] *= rng.uniform(0.0, 2.0, n).astype(np.float32)
        pos[rng.choice(n, n // 50, replace=False), 3] = 0.0   # massless tracers
    acc = _forces(pos)
    assert np.all(acc[:, 3] == 0.0) and np.all(np.isfinite(acc))
    tg = np.unique(np.concatenate([np.arange(min(n, 300)), np.arange(max(0, n - 300), n),
                                   np.random.default_rng(1).choice(n, min(n, 600))]))
    r = _rel(acc[tg, :3].astype(np.float64), O.allpairs_f64(pos, EPS, targets=tg))
    # the bounds the tiled kernel is held to (test_gpu_forces.py)
    assert np.median(r) < 2e-6 and np.percentile(r, 99) < 2e-5


@pytest.mark.parametrize("n", [2500, 9000])
@pytest.mark.parametrize("scale,mass", [(1e12, 1e30), (1e-10, 1e-6), (1e15, 1e33)])
def test_scales(n, scale, mass):
    """The factor m / r^3 is built as (m / r) / r^2, so that lengths and
    masses far from 1 keep their digits (r^-3 alone would underflow)."""
    base, _ = ic.two_disks(n, seed=3)
    pos = base.copy()
    pos[:, :3] *= np.float32(scale)
    pos[:, 3] *= np.float32(mass)
    acc = _forces(pos, eps=EPS * scale)
    r = _rel(acc[:, :3].astype(np.float64), O.allpairs_f64(pos, EPS * scale))
    assert np.median(r) < 2e-6 and np.percentile(r, 99) < 2e-5


def test_batches_and_small_scratch_give_the_same_bits():
    """Alone (whole table), in an ensemble, and in a server whose scratch
    holds a few rows of tiles at a time."""
    states = [ic.two_disks(n, seed=n) for n in (2500, 9000, 5000)]
    prm = api.SimParams(dt=0.005, epsilon=EPS, force="naive")
    alone = []
    for pos, vel in states:
        with api.Simulation(pos, vel, prm) as sim:
            sim.step(3)
            alone.append((sim.positions(), sim.velocities()))
    with Ensemble(states, prm) as ens:
        ens.step(3)
        for s, (p, v) in enumerate(alone):
            q, w = ens.state(s)
            assert np.array_equal(q, p) and np.array_equal(w, v)
    with Server(hbm_budget_bytes=24 << 20, max_sims=4) as srv:
        ids = [srv.submit(pos, vel, prm, 3) for pos, vel in states]
        for rid, (p, v) in zip(ids, alone):
            srv.wait(rid, 120)
            q, w = srv.result(rid)
            assert np.array_equal(q, p) and np.array_equal(w, v)


@pytest.mark.parametrize("n", [1000, 2559, 2560, 9000])
def test_forces_over_the_positions(n):
    """nb_compute_forces_dev with one buffer for positions and forces: each
    target's force comes from the positions, none from forces already written."""
    import ctypes

    import torch

    from nbodyssey_b200 import _lib as L
    lib = L.load()
    pos, _ = ic.two_disks(n, seed=n)
    buf = torch.from_numpy(pos).cuda()
    prm = api.SimParams(epsilon=EPS, force="naive").to_c()
    ws = ctypes.c_void_p()
    L.check(lib.nb_workspace_create(ctypes.byref(ws)))
    try:
        ptr = ctypes.c_void_p(buf.data_ptr())
        L.check(lib.nb_compute_forces_dev(ws, n, ptr, ptr, ctypes.byref(prm),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        acc = buf.cpu().numpy()
    finally:
        L.check(lib.nb_workspace_destroy(ws))
    r = _rel(acc[:, :3].astype(np.float64), O.allpairs_f64(pos, EPS))
    assert np.median(r) < 2e-6 and np.percentile(r, 99) < 2e-5
