"""The launchers captured into a caller's graph: plain edges (code that reads the
graph without edge data still can), and replays that give the bits of direct
calls."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import NativeState, Params, make_params, ptr
from .helpers import random_case
from .test_gpu_launch_errors import cudart

pytestmark = pytest.mark.gpu


def _captured(torch, call):
    """Instantiates what call(stream) launches; returns replay(), after checking the edges."""
    rt = cudart()
    stream, graph, run = torch.cuda.Stream(), C.c_void_p(), C.c_void_p()
    handle = C.c_void_p(stream.cuda_stream)
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(handle, 2) == 0
    call(handle)
    assert rt.cudaStreamEndCapture(handle, C.byref(graph)) == 0
    nodes, edges = C.c_size_t(), C.c_size_t(64)
    assert rt.cudaGraphGetNodes(graph, None, C.byref(nodes)) == 0
    a, b = (C.c_void_p * 64)(), (C.c_void_p * 64)()
    assert rt.cudaGraphGetEdges(graph, a, b, None, C.byref(edges)) == 0
    assert edges.value == nodes.value - 1 >= 1
    assert rt.cudaGraphInstantiate(C.byref(run), graph, C.c_ulonglong(0)) == 0
    assert rt.cudaGraphDestroy(graph) == 0

    def replay():
        assert rt.cudaGraphLaunch(run, handle) == 0
        assert rt.cudaStreamSynchronize(handle) == 0

    return replay


@pytest.mark.parametrize("mode,dims", [("single", (64, 20, 12)), ("single", (61, 20, 12)), ("two", (61, 20, 12))])
def test_native_steps(cuda, mode, dims):
    torch, L, (nx, ny, nz) = cuda, fg.lib(), dims
    codes, specs, rp, sources, consts, jz = random_case(*dims, seed=2, ncls=3, nsrc=2)
    raw = make_params(dims, consts, sources, jz)
    plan = fg.Plan(Params(raw), specs, scheme=fg.SCHEME_CORRECTED, rp=rp)
    states = [NativeState(torch, (nz, ny, nx), codes) for _ in range(2)]

    def steps(st, stream, n0):
        for n in (n0, n0 + 1):
            f = st.fields(n, mode == "single")
            if mode == "single":
                fg.check(L.fdtd_step(plan.handle, C.byref(f), n, stream), "fdtd_step")
            else:
                fg.check(L.fdtd_step_h(plan.handle, C.byref(f), stream), "fdtd_step_h")
                fg.check(L.fdtd_step_de(plan.handle, C.byref(f), n, stream), "fdtd_step_de")

    for st in states:
        steps(st, None, 0)
    torch.cuda.synchronize()
    replay = _captured(torch, lambda s: steps(states[0], s, 2))
    for _ in range(3):
        replay()
        steps(states[1], None, 2)
    torch.cuda.synchronize()
    got, want = (st.latest(2, mode == "single") for st in states)
    plan.close()
    assert np.any(want["ez"])
    for name in want:
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name


def test_compat_launchers(cuda):
    torch, L, dims = cuda, fg.lib(), (61, 20, 12)
    _, _, rp, sources, consts, jz = random_case(*dims, seed=3, ncls=2, nsrc=2)
    fg.check(L.fdtd_copy_symbols(C.byref(make_params(dims, consts, sources, jz))), "fdtd_copy_symbols")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    fields = [torch.randn(dims[::-1], generator=gen, device="cuda") for _ in range(21)]
    cells = [torch.rand(dims[::-1], generator=gen, device="cuda") + 1.0 for _ in range(4)]
    media = [ptr(v) for v in cells]
    keep = [torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in rp]
    slabs = [ptr(v) for v in keep]
    both = [[v.clone() for v in fields] for _ in range(2)]

    def step(v, s):
        h, e0, e1, e2, d0, d1, d2 = ([ptr(t) for t in v[3 * k:3 * k + 3]] for k in range(7))
        fg.check(L.fdtd_update_h(*h, *e2, s))
        fg.check(L.fdtd_update_d(*d0, *d2, *h, s))
        fg.check(L.fdtd_update_sources(d0[2], d2[2], h[0], h[1], 3, s))
        fg.check(L.fdtd_update_e(*e0, *e2, *e1, *d0, *d2, *d1, *media, s))
        fg.check(L.fdtd_update_mur(*e0, *e2, *slabs, s))

    replay = _captured(torch, lambda s: step(both[0], s))
    for _ in range(3):
        replay()
        step(both[1], None)
    torch.cuda.synchronize()
    for k, (got, want) in enumerate(zip(*both)):
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)), k
