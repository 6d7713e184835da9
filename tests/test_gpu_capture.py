"""The first FP64 call of a space under a relaxed capture, on a blocking and on
a non-blocking stream: it allocates its scratch, and nothing of it may touch the
legacy stream (refused while a blocking stream is captured).  The replayed graph
(FP64-pipe products, channel tiles) against the same call outside a capture
(digit products, descriptors): two FP64 sums of at most 100 terms, 1e-13 of the
largest element."""
import ctypes
import subprocess
import sys

import numpy as np
import pytest

import imsrg_gb300 as ig

pytestmark = pytest.mark.gpu


def cudart():
    rt = ctypes.CDLL("libcudart.so.13")
    rt.cudaStreamBeginCapture.argtypes = [ctypes.c_void_p, ctypes.c_int]
    rt.cudaStreamEndCapture.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_void_p)]
    rt.cudaGraphInstantiate.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_void_p, ctypes.c_ulonglong]
    rt.cudaGraphLaunch.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    rt.cudaStreamSynchronize.argtypes = [ctypes.c_void_p]
    return rt


def first_call_captured(term, nonblocking):
    rt = cudart()
    space = ig.ModelSpace(3, "O16", "O16")

    def call(dX, dY, dZ, stream):
        if term == "commutator":
            ig.Commutator.device_commutator(dX, dY, dZ, "fp64", stream)
        else:
            ig.Commutator.device_term(term, dX, dY, dZ, "fp64", stream)

    with ig.DeviceOperator(space, 1) as dX, ig.DeviceOperator(space, -1) as dY, ig.DeviceOperator(space, 1) as dZ:
        dX.fill_random(1)
        dY.fill_random(2)
        dZ.zero()
        st, graph, exe = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(st), nonblocking) == 0
        assert rt.cudaDeviceSynchronize() == 0
        assert rt.cudaStreamBeginCapture(st, 2) == 0
        try:
            call(dX, dY, dZ, st.value)
        finally:
            ended = rt.cudaStreamEndCapture(st, ctypes.byref(graph))
        assert ended == 0 and rt.cudaGraphInstantiate(ctypes.byref(exe), graph, 0) == 0
        assert rt.cudaGraphLaunch(exe, st) == 0 and rt.cudaStreamSynchronize(st) == 0
        got = dZ.download()
        dZ.zero()
        call(dX, dY, dZ, None)
        want = dZ.download()
    assert np.linalg.norm(want) > 0
    assert np.max(abs(got - want)) <= 1e-13 * np.max(abs(want))


@pytest.mark.parametrize("term", ["commutator", "comm222_phss", "comm222_pp_hhss"])
@pytest.mark.parametrize("nonblocking", [0, 1])
def test_first_call_under_capture(term, nonblocking, monkeypatch):
    # (a process each: a refused capture leaves its error for the next call)
    monkeypatch.setenv("IMSRG_GB300_TUNING", "off")
    code = "import sys; sys.path[:0] = ['.', 'tests']; import test_gpu_capture as t; t.first_call_captured(%r, %d)"
    r = subprocess.run([sys.executable, "-c", code % (term, nonblocking)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
