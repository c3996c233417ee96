"""Handles, workspaces and batches of different sizes side by side: a call's
launch depends on nothing that another thread's call, or this thread's call on
another handle, has set before."""
import ctypes
import threading

import numpy as np
import pytest

from nbodyssey_b200 import _lib as L
from nbodyssey_b200 import api, ic
from nbodyssey_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu
PRM = api.SimParams(dt=0.005, epsilon=0.05, force="naive")


def _run(workers):
    """Runs the callables in threads, started together; their exceptions."""
    gate, errors = threading.Barrier(len(workers)), []

    def body(fn):
        gate.wait()
        try:
            fn()
        except Exception as e:   # noqa: BLE001 - reported below
            errors.append(e)

    th = [threading.Thread(target=body, args=(w,)) for w in workers]
    for t in th:
        t.start()
    for t in th:
        t.join()
    return errors


def _device_forces(n, calls, out):
    import torch
    lib = L.load()
    pos, _ = ic.two_disks(n, seed=n)
    d_pos = torch.from_numpy(pos).cuda()
    d_acc = torch.zeros_like(d_pos)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    prm = PRM.to_c()
    ws = ctypes.c_void_p()
    L.check(lib.nb_workspace_create(ctypes.byref(ws)))

    def call():
        L.check(lib.nb_compute_forces_dev(ws, n, ctypes.c_void_p(d_pos.data_ptr()),
                                          ctypes.c_void_p(d_acc.data_ptr()), ctypes.byref(prm),
                                          ctypes.c_void_p(stream.cuda_stream)))

    def work():
        try:
            for k in range(calls):
                call()
                if k % 16 == 15:
                    stream.synchronize()
        finally:
            stream.synchronize()
            out[n] = d_acc.cpu().numpy()
            L.check(lib.nb_workspace_destroy(ws))

    call()
    stream.synchronize()
    out["alone", n] = d_acc.cpu().numpy()
    return work


def test_all_pairs_of_two_sizes_from_two_threads():
    out = {}
    sizes = (3000, 200_000)
    errors = _run([_device_forces(3000, 20_000, out), _device_forces(200_000, 300, out)])
    assert not errors, errors
    for n in sizes:
        assert np.array_equal(out[n], out["alone", n]), n


def test_all_pairs_batches_of_two_sizes_from_two_threads():
    small = [ic.two_disks(n, seed=n) for n in (2600, 3000)]
    large = [ic.two_disks(n, seed=n) for n in (70_000, 2700)]
    ref = {}
    for name, states in (("small", small), ("large", large)):
        with Ensemble(states, PRM) as e:
            e.set_graphs(False)
            e.step(40)
            ref[name] = [e.state(s) for s in range(len(states))]
    got = {}

    def work(name, states, rounds):
        def go():
            for _ in range(rounds):
                with Ensemble(states, PRM) as e:
                    e.set_graphs(False)
                    e.step(40)
                    got[name] = [e.state(s) for s in range(len(states))]
        return go

    errors = _run([work("small", small, 60), work("large", large, 6)])
    assert not errors, errors
    for name in ref:
        for (p, v), (q, w) in zip(ref[name], got[name]):
            assert np.array_equal(p, q) and np.array_equal(v, w), name


def test_captured_step_after_a_call_of_another_size():
    pos, vel = ic.two_disks(200_000, seed=5)
    with api.Simulation(pos, vel, PRM) as sim:
        sim.step(3)
        ref = sim.positions()
    other, _ = ic.two_disks(3000, seed=6)
    with api.Simulation(pos, vel, PRM) as sim, \
            api.Simulation(other, np.zeros_like(other), PRM) as small:
        for _ in range(3):
            sim.step(1)
            small.compute_forces()
        assert np.array_equal(sim.positions(), ref)
