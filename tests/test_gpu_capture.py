"""Sweeps recorded by a stream capture of the context's stream: nothing is allocated or timed on the way,
and the replayed graph sweeps the same chain as the call."""
import ctypes as C

import numpy as np
import pytest

from nanomagmc_gb300 import _lib as L
from test_gpu_sequenced import CASES, sampler

pytestmark = pytest.mark.gpu


def check(rc):
    assert rc == 0, rc


@pytest.mark.parametrize("name", ["four_site", "odd_rows", "ising_words", "classes", "colours"])
def test_captured_sweeps(tmp_path, name):
    rt = C.CDLL("libcudart.so")
    a, b = sampler(tmp_path, CASES[name], 3), sampler(tmp_path, CASES[name], 3)
    a.measure()   # the points are on the device
    b.measure()
    graph, ex = C.c_void_p(), C.c_void_p()
    stream = C.c_void_p(a.stream())
    check(rt.cudaStreamBeginCapture(stream, 1))   # this thread
    a.sweep(2)
    check(rt.cudaStreamEndCapture(stream, C.byref(graph)))
    check(rt.cudaGraphInstantiate(C.byref(ex), graph, C.c_ulonglong(0)))
    for _ in range(3):
        check(rt.cudaGraphLaunch(ex, stream))
    a.synchronize()
    b.sweep(6)
    for k in range(3):
        assert np.array_equal(a.get_spins(k), b.get_spins(k))
    check(rt.cudaGraphExecDestroy(ex))
    check(rt.cudaGraphDestroy(graph))
    a.sweep(1)   # the class planes are taken up now
    b.sweep(1)
    for k in range(3):
        assert np.array_equal(a.get_spins(k), b.get_spins(k))
    a.close()
    b.close()


@pytest.mark.parametrize("name", ["four_site", "ising_words", "ising", "classes"])
def test_points_changed_between_replays(tmp_path, name):
    """A graph of sweeps follows points that are uploaded after it was recorded."""
    rt = C.CDLL("libcudart.so")
    a, b = sampler(tmp_path, CASES[name], 3), sampler(tmp_path, CASES[name], 3)
    for s in (a, b):
        s.sweep(1)
        s.measure()
    graph, ex = C.c_void_p(), C.c_void_p()
    stream = C.c_void_p(a.stream())
    check(rt.cudaStreamBeginCapture(stream, 1))
    a.sweep(2)
    check(rt.cudaStreamEndCapture(stream, C.byref(graph)))
    check(rt.cudaGraphInstantiate(C.byref(ex), graph, C.c_ulonglong(0)))
    for T in (0.7, 3.0, 1.1):
        for s in (a, b):
            s.set_points(np.arange(3), np.full(3, T), np.linspace(0.4, -0.4, 3))
            s.measure()   # uploads them
        check(rt.cudaGraphLaunch(ex, stream))
        a.synchronize()
        b.sweep(2)
        for k in range(3):
            assert np.array_equal(a.get_spins(k), b.get_spins(k))
    check(rt.cudaGraphExecDestroy(ex))
    check(rt.cudaGraphDestroy(graph))
    a.close()
    b.close()
