"""The server's all-pairs scratch pool: what is admitted and what runs
side by side follow from the least region a request can run with."""
import ctypes

import numpy as np
import pytest

from nbodyssey_b200 import _lib as L
from nbodyssey_b200 import api, ic
from nbodyssey_b200.server import Server

pytestmark = pytest.mark.gpu
PRM = api.SimParams(dt=0.005, epsilon=0.05, force="naive")


@pytest.fixture
def table():
    """A tuning table to change; the one before is put back."""
    base = api.tune_get()
    yield dict(base)
    api.tune_set(base)


def _alone(pos, vel, steps):
    with api.Simulation(pos, vel, PRM) as sim:
        sim.step(steps)
        return sim.positions(), sim.velocities()


@pytest.mark.parametrize("n", [17_001, 20_001, 70_001])
def test_a_region_smaller_than_one_row_of_tiles(table, n):
    """With one source chunk per target tile the least region is the packed
    sources' (n float4), a third of one row of tiles; the budget is the least
    that holds the particles."""
    table["ap_ctas"] = [1] * L.NB_TUNE_BUCKETS
    api.tune_set(table)
    pos, vel = ic.two_disks(n, seed=9)
    slots = (n + 4095) // 4096 * 4096
    with Server(hbm_budget_bytes=slots * 232 * 8 // 7 + 4096, max_sims=2) as srv:
        rid = srv.submit(pos, vel, PRM, 3)
        srv.wait(rid, 120)
        p, v = srv.result(rid)
    q, w = _alone(pos, vel, 3)
    assert np.array_equal(p, q) and np.array_equal(v, w)


def test_whole_tables_do_not_keep_requests_out(table):
    """150 requests of 2,560 particles: their least regions (16 units of 16 KiB
    with the default shapes) fit the pool of 3,200 units, their whole tables (50)
    do not."""
    t = L.nb_tune_table()
    L.check(L.load().nb_tune_defaults(ctypes.byref(t)))
    table["ap_threads"], table["ap_k"] = list(t.ap_threads), list(t.ap_k)
    table["ap_ctas"] = list(t.ap_ctas)
    api.tune_set(table)
    states = [ic.two_disks(2560, seed=k) for k in range(4)]
    steps = 2500
    with Server(hbm_budget_bytes=3200 * 16384 * 8, max_sims=256) as srv:
        ids = [srv.submit(*states[k % 4], PRM, steps) for k in range(150)]
        for rid in ids:
            srv.wait(rid, 120)
        peak = srv.stats()["peak_running"]
        got = [srv.result(rid) for rid in ids]
    assert peak == 150
    for k, (pos, vel) in enumerate(states):
        q, w = _alone(pos, vel, steps)
        for p, v in got[k::4]:
            assert np.array_equal(p, q) and np.array_equal(v, w)


def test_regions_move_as_requests_come_and_go(table):
    """Requests of all three all-pairs kernels and of different lengths over a pool
    that cannot hold their whole tables: each one's region grows, shrinks and moves
    between steps (the second packed one when the first has gone)."""
    t = L.nb_tune_table()
    L.check(L.load().nb_tune_defaults(ctypes.byref(t)))
    L.check(L.load().nb_tune_set(ctypes.byref(t)))
    work = [((1 << 20) + 1, 1), ((1 << 20) + 31, 3), (70_001, 5), (9000, 4), (20_001, 2),
            (1500, 5)]
    states = [ic.two_disks(n, seed=n) for n, _ in work]
    with Server(hbm_budget_bytes=1 << 30, max_sims=8) as srv:
        ids = [srv.submit(*s, PRM, k) for s, (_, k) in zip(states, work)]
        got = []
        for rid in ids:
            srv.wait(rid, 120)
            got.append(srv.result(rid))
    for (pos, vel), (_, k), (p, v) in zip(states, work, got):
        q, w = _alone(pos, vel, k)
        assert np.array_equal(p, q) and np.array_equal(v, w)
