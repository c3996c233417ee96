"""The tree build at the edges of its rules: leaf groups of 256, 512 or 1,024
(the fewest leaves that need no more levels than 1,024 do: 15 segments per later
CTA with 30-bit keys, 10 with 63-bit), a thread per leaf up to 1,024 leaves per
SM, and trees whose depth comes from equal keys."""
import numpy as np
import pytest

from nbodyssey_b200 import api, ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(pos, bits):
    prm = api.SimParams(epsilon=0.05, theta=0.5, force="bh", traverse="warp", key_bits=bits)
    with api.Simulation(pos, np.zeros_like(pos), prm) as sim:
        t = sim.debug_lbvh()
    o = O.Tree(pos, bits)
    assert np.array_equal(t["children"], o.children)
    assert np.array_equal(t["parent"], o.parent)
    assert np.array_equal(t["com4"], o.com)
    assert np.array_equal(t["size2"], o.size2)


@pytest.mark.parametrize("n,bits", [
    (255, 30), (256, 30), (257, 30), (511, 30), (513, 63), (3840, 30), (3841, 30),
    (15_360, 30), (15_361, 30), (57_600, 30), (57_601, 30), (115_200, 30), (115_201, 30),
    (151_552, 30), (151_553, 30), (230_400, 30), (230_401, 30),
    (2560, 63), (2561, 63), (10_240, 63), (10_241, 63), (25_600, 63), (25_601, 63),
    (102_400, 63), (102_401, 63)])
def test_group_edges(n, bits):
    pos, _ = ic.two_disks(n, seed=n)
    _check(pos, bits)


@pytest.mark.parametrize("n", [2000, 20_000, 60_000])
def test_equal_keys(n):
    """Coincident runs longer than a group: splits decided by the index."""
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.normal(size=(n, 3)).astype(np.float32)
    pos[n // 4: n // 2, :3] = pos[0, :3]
    pos[n // 2: n // 2 + 700, :3] = pos[1, :3]
    pos[:, 3] = 1.0 / n
    _check(pos, 30)
