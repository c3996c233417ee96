"""Energy diagnostic (src/integrator.cu:43-110) at the tile edges of its
kernels: tiles of 128 particles below n = 16,384, of 512 from there, partners
in stages of 256."""
import numpy as np
import pytest

from nbodyssey_b200 import api, ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EPS = 0.05


@pytest.mark.parametrize("n", [1, 2, 3, 127, 128, 129, 255, 256, 257, 513, 1025,
                               16383, 16384, 16385, 20011])
def test_energy_vs_fp64(n):
    pos, vel = ic.two_disks(max(n, 2), seed=n)
    pos, vel = pos[:n], vel[:n]
    with api.Simulation(pos, vel, api.SimParams(epsilon=EPS, force="naive")) as sim:
        e, ke, pe = sim.energy()
    ref = O.energy_f64(pos, vel, EPS)
    m = pos[:, 3].astype(np.float64)
    # PE = -1/2 sum_i m_i phi_i: each FP32 term is within 2^-22 (approximate
    # rsqrt) + 3 2^-24 (r^2), each FP32 sum of at most 256 terms within
    # 256 2^-24, of phi_i plus the self term m_i / eps it carries
    rel = 2.0 ** -22 + 259 * 2.0 ** -24
    size = abs(ref[2]) + 0.5 * np.sum(m * m) / EPS
    assert abs(pe - ref[2]) <= rel * size
    assert abs(ke - ref[1]) <= 1e-12 * abs(ref[1])
    assert abs(e - (ke + pe)) <= 1e-12 * (abs(ke) + abs(pe))
    if n == 1:
        assert pe == 0.0


@pytest.mark.parametrize("eps", [0.05, 1e-4])
@pytest.mark.parametrize("n,where", [(129, 0), (513, 512), (1000, 500), (2560, 2559),
                                     (16384, 8192), (20011, 20010)])
def test_energy_with_a_dominant_body(n, where, eps):
    """A central body of 10^6 times the others' mass: its self term would be far
    larger than the sum of the others' terms in its potential."""
    pos, vel = ic.two_disks(n, seed=n)
    pos[where, 3] *= np.float32(1e6)
    with api.Simulation(pos, vel, api.SimParams(epsilon=eps, force="naive")) as sim:
        _, _, pe = sim.energy()
    ref = O.energy_f64(pos, vel, eps)[2]
    # as above, but every FP32 sum holds terms of the potential alone; close
    # pairs at small eps: each r^2 is of differences exact to 2^-24 of themselves
    rel = 2.0 ** -22 + 259 * 2.0 ** -24
    assert abs(pe - ref) <= rel * abs(ref)
