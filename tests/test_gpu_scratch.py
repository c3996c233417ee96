"""All-pairs scratch: calls under stream capture on a workspace that has been
used before, tables that cannot be had, and captured steps whose scratch moves."""
import ctypes

import numpy as np
import pytest

from nbodyssey_b200 import _lib as L
from nbodyssey_b200 import api, ic
from nbodyssey_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu
EPS = 0.05
PRM = api.SimParams(dt=0.005, epsilon=EPS, force="naive")


class _Dev:
    """A device-pointer caller: a workspace and the arrays of one size."""

    def __init__(self):
        self.lib = L.load()
        self.ws = ctypes.c_void_p()
        L.check(self.lib.nb_workspace_create(ctypes.byref(self.ws)))

    def close(self):
        L.check(self.lib.nb_workspace_destroy(self.ws))

    def forces(self, pos, acc):
        import torch
        L.check(self.lib.nb_compute_forces_dev(
            self.ws, pos.shape[0], ctypes.c_void_p(pos.data_ptr()),
            ctypes.c_void_p(acc.data_ptr()), ctypes.byref(PRM.to_c()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


def _captured(fn):
    import torch
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        fn()
    graph.replay()
    torch.cuda.synchronize()


# each size starts a range of larger tiles, whose whole table is smaller than
# the one of the size below it
@pytest.mark.parametrize("n", [16_384, 24_576, 65_536])
def test_capture_of_a_smaller_call_than_the_warm_up(n):
    import torch
    dev = _Dev()
    try:
        first = torch.from_numpy(ic.two_disks(n + 1, seed=1)[0]).cuda()
        dev.forces(first, torch.zeros_like(first))
        pos = torch.from_numpy(ic.two_disks(n, seed=2)[0]).cuda()
        acc = torch.zeros_like(pos)
        _captured(lambda: dev.forces(pos, acc))
        got = acc.cpu().numpy()
        dev.forces(pos, acc)
        assert np.array_equal(got, acc.cpu().numpy())
    finally:
        dev.close()


@pytest.mark.parametrize("n", [16_384, 24_576, 65_536, 163_840])
def test_scratch_grows_only_with_n(n):
    import torch
    dev, fresh = _Dev(), _Dev()
    try:
        first = torch.from_numpy(ic.two_disks(n + 1, seed=1)[0]).cuda()
        dev.forces(first, torch.zeros_like(first))
        pos = torch.from_numpy(ic.two_disks(n, seed=2)[0]).cuda()
        acc, ref = torch.zeros_like(pos), torch.zeros_like(pos)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        dev.forces(pos, acc)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
        fresh.forces(pos, ref)
        assert torch.equal(acc, ref)
    finally:
        dev.close()
        fresh.close()


def test_capture_of_a_larger_call_than_the_warm_up_is_refused():
    """As any capture that would have to allocate; the workspace stays usable."""
    import torch
    dev = _Dev()
    try:
        first = torch.from_numpy(ic.two_disks(5000, seed=1)[0]).cuda()
        acc = torch.zeros_like(first)
        dev.forces(first, acc)
        ref = acc.cpu().numpy()
        pos = torch.from_numpy(ic.two_disks(50_000, seed=2)[0]).cuda()
        out = torch.zeros_like(pos)
        with pytest.raises(Exception):
            _captured(lambda: dev.forces(pos, out))
        dev.forces(first, acc)
        assert np.array_equal(acc.cpu().numpy(), ref)
    finally:
        dev.close()


@pytest.mark.parametrize("n", [1, 1000, 2559, 2560, 9000, 60_001])
def test_capture_of_forces_over_the_positions_after_a_warm_up_beside_them(n):
    import torch
    dev = _Dev()
    try:
        pos = torch.from_numpy(ic.two_disks(max(n, 2), seed=3)[0][:n]).cuda()
        acc = torch.zeros_like(pos)
        dev.forces(pos, acc)
        buf = pos.clone()
        _captured(lambda: dev.forces(buf, buf))
        assert np.array_equal(buf.cpu().numpy(), acc.cpu().numpy())
    finally:
        dev.close()


# rows of tiles at a time (8 MiB) and chunks of one row (1 MiB) of a table of 38
@pytest.mark.parametrize("mib", ["8", "1"])
def test_table_that_cannot_be_had(monkeypatch, mib):
    """A table refused (here by the limit) is done without: the same bits from a
    smaller one, eagerly, through the step graph and under capture, and nothing
    changes for the handle once there is room again."""
    import torch
    n = 20_001
    pos, vel = ic.two_disks(n, seed=4)
    with api.Simulation(pos, vel, PRM) as sim:
        ref = sim.compute_forces()
        sim.step(3)
        end = sim.positions()
    monkeypatch.setenv("NBODY_B200_ALLPAIRS_MIB", mib)
    with api.Simulation(pos, vel, PRM) as sim:
        for _ in range(2):
            assert np.array_equal(sim.compute_forces(), ref)
        sim.step(1)
        sim.compute_forces()
        sim.step(1)
        monkeypatch.delenv("NBODY_B200_ALLPAIRS_MIB")
        sim.compute_forces()
        sim.step(1)
        assert np.array_equal(sim.positions(), end)
    monkeypatch.setenv("NBODY_B200_ALLPAIRS_MIB", mib)
    dev = _Dev()
    try:
        d_pos = torch.from_numpy(pos).cuda()
        acc = torch.zeros_like(d_pos)
        dev.forces(d_pos, acc)
        acc.zero_()
        _captured(lambda: dev.forces(d_pos, acc))
        assert np.array_equal(acc.cpu().numpy(), ref)
        buf = d_pos.clone()
        dev.forces(buf, buf)   # the copy of the positions beside such a table
        assert np.array_equal(buf.cpu().numpy(), ref)
    finally:
        dev.close()


def test_limit_bounds_the_memory_of_a_handle(monkeypatch):
    """Without it 262,144 particles take 0.8 GB."""
    import torch
    pos, vel = ic.two_disks(262_144, seed=5)
    with api.Simulation(pos[:64].copy(), vel[:64].copy(), PRM):   # kernels and tuning first
        pass
    monkeypatch.setenv("NBODY_B200_ALLPAIRS_MIB", "64")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with api.Simulation(pos, vel, PRM):
        assert free - torch.cuda.mem_get_info()[0] < 160 << 20


def test_step_graph_follows_scratch_that_moved():
    """Above 2^20 particles a table set by hand can ask for more partials: a
    force call then moves the scratch that the captured step uses."""
    n = (1 << 20) + 1
    pos, vel = ic.two_disks(n, seed=6)
    base = api.tune_get()
    out = []
    try:
        for graphs in (True, False):
            api.tune_set(dict(base, ap_threads=[256] * L.NB_TUNE_BUCKETS,
                              ap_k=[8] * L.NB_TUNE_BUCKETS,
                              ap_ctas=[1024] * L.NB_TUNE_BUCKETS))   # 513 tiles: 2 chunks
            with api.Simulation(pos, vel, PRM) as sim:
                sim.set_graphs(graphs)
                sim.step(1)
                api.tune_set(dict(base, ap_threads=[256] * L.NB_TUNE_BUCKETS,
                                  ap_k=[8] * L.NB_TUNE_BUCKETS,
                                  ap_ctas=[3000] * L.NB_TUNE_BUCKETS))   # 6 chunks
                sim.compute_forces()
                sim.step(1)
                out.append(sim.positions())
    finally:
        api.tune_set(base)
    assert np.array_equal(*out)


def test_batch_tables_that_cannot_be_had(monkeypatch):
    """Eight simulations of 40,000 particles take 614 MB with whole tables; where
    those cannot be had the batch is made with the least regions (160 MB with the
    default shapes), its results unchanged."""
    import ctypes as C

    import torch
    base = api.tune_get()
    t = L.nb_tune_table()
    L.check(L.load().nb_tune_defaults(C.byref(t)))
    try:
        L.check(L.load().nb_tune_set(C.byref(t)))
        states = [ic.two_disks(40_000, seed=k) for k in range(8)]
        with Ensemble(states, PRM) as ens:
            ens.step(2)
            ref = [ens.state(s) for s in range(8)]
        monkeypatch.setenv("NBODY_B200_ALLPAIRS_MIB", "256")
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        with Ensemble(states, PRM) as ens:
            assert free - torch.cuda.mem_get_info()[0] < 350 << 20
            ens.step(2)
            for s in range(8):
                p, v = ens.state(s)
                assert np.array_equal(p, ref[s][0]) and np.array_equal(v, ref[s][1])
    finally:
        api.tune_set(base)


def test_batch_above_one_gib_of_tables_takes_few_passes():
    """524,288 particles have 128 rows of tiles and tables of 3.2 GB; 1 GiB holds
    42 rows."""
    base = api.tune_get()
    t = L.nb_tune_table()
    L.check(L.load().nb_tune_defaults(ctypes.byref(t)))
    try:
        L.check(L.load().nb_tune_set(ctypes.byref(t)))
        with Ensemble([ic.two_disks(524_288, seed=3)], PRM) as ens:
            assert ens.kernels_per_step() == 1 + 2 * 4
    finally:
        api.tune_set(base)
