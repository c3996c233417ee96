"""The two sorts of the tree build against the oracle's stable sort: one
cluster launch (up to 65,536 particles, 36,864 with 63-bit keys; slices of
n / 16 rounded up to 32 keys, 512 threads) and the onesweep passes above
(2,048-key tiles up to 303,104 keys, then 4,096)."""
import numpy as np
import pytest

from nbodyssey_b200 import api, ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(pos, bits):
    prm = api.SimParams(epsilon=0.05, theta=0.5, force="bh", traverse="warp", key_bits=bits)
    with api.Simulation(pos, np.zeros_like(pos), prm) as sim:
        t = sim.debug_lbvh()
    lo, hi = O.bbox(pos)
    keys, perm = O.sort_pairs(O.morton_keys(pos, bits, lo, hi), bits)
    assert np.array_equal(t["keys"], keys)
    assert np.array_equal(t["perm"], perm)


@pytest.mark.parametrize("n", [2, 32, 33, 511, 512, 513, 16 * 512 - 1, 16 * 512, 16 * 512 + 1,
                               20_011, 36_863, 36_864, 36_865, 53_248, 53_249,
                               65_535, 65_536, 65_537, 69_632, 69_633, 303_104, 303_105,
                               307_201])
@pytest.mark.parametrize("bits", [30, 63])
def test_sizes(n, bits):
    pos, _ = ic.two_disks(n, seed=n)
    _check(pos, bits)


@pytest.mark.parametrize("n", [40_000, 70_000])
@pytest.mark.parametrize("bits", [30, 63])
def test_few_distinct_keys(n, bits):
    """Long runs of one digit, whole slices and tiles of them, stay in order;
    one axis without extent."""
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :2] = rng.integers(0, 3, (n, 2)).astype(np.float32)
    pos[: n // 3, :2] = 1.0
    pos[:, 3] = 1.0 / n
    _check(pos, bits)
