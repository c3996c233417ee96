"""All-pairs around 2^20 particles, where the pairs-once kernel (its table in
several passes from 1 GiB on) gives way to the tiled one with the shapes of the
tuning table, alone and in a batch; and the launches a batch's kernels take."""
import ctypes

import numpy as np
import pytest

from nbodyssey_b200 import _lib as L
from nbodyssey_b200 import api, ic
from nbodyssey_b200.ensemble import Ensemble
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EPS = 0.05
PRM = api.SimParams(dt=0.005, epsilon=EPS, force="naive")
TOP = 1 << 20


def _targets(n):
    rng = np.random.default_rng(n)
    return np.unique(np.concatenate([[0, 1, n - 2, n - 1], rng.choice(n, 90, replace=False)]))


def _check(pos, acc, median, tail):
    tg = _targets(len(pos))
    exact = O.allpairs_f64(pos, EPS, targets=tg)
    assert np.all(np.isfinite(acc)) and np.all(acc[:, 3] == 0.0)
    r = np.linalg.norm(acc[tg, :3] - exact, axis=1) / np.linalg.norm(exact, axis=1)
    assert np.median(r) < median and r.max() < tail


# the bounds the kernel is held to below (test_gpu_allpairs_sym.py)
@pytest.mark.parametrize("n", [400_003, TOP])
def test_pairs_once_in_several_passes(n):
    pos, vel = ic.two_disks(n, seed=n)
    with api.Simulation(pos, vel, PRM) as sim:
        _check(pos, sim.compute_forces(), 2e-6, 2e-5)


def test_closing_kick_in_several_passes(monkeypatch):
    """A step of 400,003 particles: the passes of 1 GiB and of 64 MiB give the
    same positions and velocities, and the velocities are those of the kicks."""
    pos, vel = ic.two_disks(400_003, seed=11)
    out = []
    for mib in (None, "64"):
        if mib:
            monkeypatch.setenv("NBODY_B200_ALLPAIRS_MIB", mib)
        with api.Simulation(pos, vel, PRM) as sim:
            a0 = sim.compute_forces()
            sim.step(1)
            out.append((sim.positions(), sim.velocities(), a0, sim.accelerations()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    _, v, a0, a1 = out[0]
    want = vel[:, :3] + np.float64(np.float32(0.0025)) * (a0[:, :3].astype(np.float64) + a1[:, :3])
    # two roundings to FP32, each half a unit in the last place
    size = np.maximum(np.abs(vel[:, :3]), np.abs(v[:, :3])) + 0.0025 * np.abs(a0[:, :3])
    assert np.all(np.abs(v[:, :3] - want) <= 2.0 ** -23 * size)


def test_tiled_shapes_by_hand():
    """All six launch shapes at three source chunks: the order of a target's sum
    follows from the chunks alone, so the shapes give the same bits.  Against FP64
    with a thousand massive particles among massless ones: a tile left out would
    show, and no sum has more terms than the other kernels' tests."""
    import torch
    n = TOP + 1
    pos, _ = ic.two_disks(n, seed=12)
    few = pos.copy()
    heavy = np.random.default_rng(2).choice(n, 1000, replace=False)
    few[:, 3] = 0.0
    few[heavy, 3] = 1e-3
    base = api.tune_get()
    lib = L.load()
    ws = ctypes.c_void_p()
    L.check(lib.nb_workspace_create(ctypes.byref(ws)))

    def forces(rows):
        d_pos = torch.from_numpy(rows).cuda()
        acc = torch.zeros_like(d_pos)
        L.check(lib.nb_compute_forces_dev(
            ws, n, ctypes.c_void_p(d_pos.data_ptr()), ctypes.c_void_p(acc.data_ptr()),
            ctypes.byref(PRM.to_c()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return acc.cpu().numpy()

    first = None
    try:
        for threads in (128, 256):
            for k in (2, 4, 8):
                tiles = -(-n // (threads * k))
                api.tune_set(dict(base, ap_threads=[threads] * L.NB_TUNE_BUCKETS,
                                  ap_k=[k] * L.NB_TUNE_BUCKETS,
                                  ap_ctas=[3 * tiles] * L.NB_TUNE_BUCKETS))
                _check(few, forces(few), 2e-6, 2e-5)
                acc = forces(pos)
                if first is None:
                    first = acc
                assert np.array_equal(acc, first), (threads, k)
    finally:
        api.tune_set(base)
        L.check(lib.nb_workspace_destroy(ws))


def test_batch_with_a_member_above_the_pairs_once_kernel():
    """The tiled kernel's work queue beside the other two, a Barnes-Hut member
    in the tree pipeline: each as alone."""
    states = [ic.two_disks(n, seed=20 + k) for k, n in enumerate((1000, TOP + 1, 9000, 5000))]
    params = [api.SimParams(dt=0.005, epsilon=EPS, force=f)
              for f in ("naive", "naive", "naive", "bh")]
    with Ensemble(states, params) as ens:
        ens.step(1)
        got = [(*ens.state(s), ens.accelerations(s)) for s in range(4)]
    for (pos, vel), prm, g in zip(states, params, got):
        with api.Simulation(pos, vel, prm) as sim:
            sim.step(1)
            for a, b in zip(g, (sim.positions(), sim.velocities(), sim.accelerations())):
                assert np.array_equal(a, b), len(pos)


def test_launches_of_the_all_pairs_kernels_in_a_batch():
    """Prep; one launch for all members below 2,560 particles; two (pairs and
    their sums) for all others."""
    def count(*sizes):
        with Ensemble([ic.two_disks(n, seed=n) for n in sizes], PRM) as ens:
            return ens.kernels_per_step()
    assert count(1000) == 2 and count(64, 1000, 2559) == 2
    assert count(2560, 9000) == 3 and count(1000, 2560, 20_000) == 4
