"""All-pairs scratch: calls under stream capture on a workspace that has been
used before."""
import ctypes

import numpy as np
import pytest

from nbodyssey_b200 import _lib as L
from nbodyssey_b200 import api, ic

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
