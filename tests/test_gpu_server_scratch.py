"""The server's all-pairs scratch pool: what is admitted follows from
the least region a request can run with."""
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
