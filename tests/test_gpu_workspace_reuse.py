"""A workspace reserved for many particles builds the trees of fewer: sizes whose
first level has the most groups (full later levels, 256 leaves a group)."""
import ctypes

import numpy as np
import pytest

from nbodyssey_b200 import _lib as L
from nbodyssey_b200 import api, ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap,bits,sizes", [
    (1_000_000, 30, (864_000, 57_600, 3840)),
    (300_000, 63, (256_000, 25_600, 57_600)),
])
def test_smaller_trees_in_a_larger_workspace(cap, bits, sizes):
    import torch
    lib = L.load()
    pos = torch.from_numpy(ic.two_disks(cap, seed=8)[0]).cuda()
    out = {}

    def forces(ws, n, kb):
        acc = torch.zeros_like(pos[:n])
        prm = api.SimParams(epsilon=0.05, theta=0.7, force="bh", traverse="warp", key_bits=kb)
        L.check(lib.nb_compute_forces_dev(
            ws, n, ctypes.c_void_p(pos.data_ptr()), ctypes.c_void_p(acc.data_ptr()),
            ctypes.byref(prm.to_c()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return acc.cpu().numpy()

    big = ctypes.c_void_p()
    L.check(lib.nb_workspace_create(ctypes.byref(big)))
    try:
        forces(big, cap, bits)
        for n in sizes:
            for kb in {30, bits}:
                out[n, kb] = forces(big, n, kb)
    finally:
        L.check(lib.nb_workspace_destroy(big))
    for (n, kb), got in out.items():
        ws = ctypes.c_void_p()
        L.check(lib.nb_workspace_create(ctypes.byref(ws)))
        try:
            assert np.array_equal(got, forces(ws, n, kb)), (n, kb)
        finally:
            L.check(lib.nb_workspace_destroy(ws))
