"""A handle's first reconstruction beside another stream's capture: the library
works on its own stream and touches no other, so a capture under way on a
stream that waits for the default one (a blocking stream) goes on."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W
from mprw.model import ACTIVE

RELAXED = 2   # cudaStreamCaptureModeRelaxed: allocations allowed meanwhile


def _reconstruct():
    g, f, p, opt = W.uniform_pulse(n_particles=500)
    p.cell = (5 + np.arange(p.n) % 60).astype(np.int32)
    p.status[:] = ACTIVE
    with mprw.Tracker(g, opt) as tr:
        tr.set_particles(p)
        return tr.gpkde((200.0, 1.0, 1.0), (1.0, 1.0, 1.0))[0]


def test_first_reconstruction_beside_a_capture(gpu_lib):
    want = _reconstruct()
    rt = ctypes.CDLL("libcudart.so.13")
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, RELAXED) == 0
    try:
        got = _reconstruct()
    finally:
        ended = rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
        rt.cudaGetLastError()
        if graph:
            rt.cudaGraphDestroy(graph)
        rt.cudaStreamDestroy(stream)
    assert ended == 0 and graph.value
    np.testing.assert_array_equal(got, want)
