"""A launcher that fails reports its error once: later calls, of this library
or of another one that asks CUDA for the last error, start clean."""
from __future__ import annotations

import ctypes as C

import pytest

import fdtd_gb300 as fg

from .gpu_util import make_params, ptr, zeros
from .helpers import random_case

pytestmark = pytest.mark.gpu


def cudart():
    """The CUDA runtime that torch and the library have loaded."""
    fg.lib()
    path = next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line)
    return C.CDLL(path)


def test_a_refused_launch_leaves_no_error_behind(cuda):
    torch, L, rt = cuda, fg.lib(), cudart()
    dims = (17, 9, 6)
    _, _, _, sources, consts, jz = random_case(*dims, seed=1, ncls=2, nsrc=1)
    fg.check(L.fdtd_copy_symbols(C.byref(make_params(dims, consts, sources, jz))), "fdtd_copy_symbols")
    buf = [ptr(zeros(torch, dims[::-1])) for _ in range(6)]
    torch.cuda.synchronize()
    assert rt.cudaPeekAtLastError() == 0
    # the legacy stream takes no launch while another stream of the device is being captured
    stream, graph = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 0) == 0
    status = L.fdtd_update_h(*buf, None)
    left = rt.cudaPeekAtLastError()
    rt.cudaStreamEndCapture(stream, C.byref(graph))
    rt.cudaGetLastError()
    rt.cudaStreamDestroy(stream)
    assert status != 0
    assert left == 0
    assert L.fdtd_update_h(*buf, None) == 0
    torch.cuda.synchronize()
