"""Class bytes beyond the caller's table.  A single-pass step takes the table's
last class for them on every route: the z-marching kernel (addressable rows)
and the two-pass kernels (rows or bases that TMA cannot address), with a plan's
table and with the static entry point's.  fdtd_step_de has a table of all 256
rows, those without a class zero, and E is 0 on such cells."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import NativeState, Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu

NCLS, STEPS = 3, 6


def _case(dims):
    codes, specs, rp, sources, consts, jz = random_case(*dims, seed=sum(dims), ncls=NCLS, nsrc=2)
    beyond = codes.copy()
    cells = np.flatnonzero(codes == NCLS - 1)
    beyond.flat[cells] = np.resize(np.array([NCLS, 63, 64, 71, 72, 200, 255], np.uint8), cells.size)
    return codes, beyond, specs, rp, make_params(dims, consts, sources, jz)


def _run(torch, dims, raw, codes, specs, rp, static, shift):
    nx, ny, nz = dims
    st = NativeState(torch, (nz, ny, nx), codes)
    if shift:
        for slot in [v for slots in (st.h, st.e, st.d) for v in slots]:
            for k in range(3):
                big = torch.zeros(slot[k].numel() + 4, device="cuda")
                slot[k] = big[shift:shift + slot[k].numel()].view(slot[k].shape)
    plan = None if static else fg.Plan(Params(raw), specs, scheme=fg.SCHEME_CORRECTED, rp=rp)
    slabs = [torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in rp]
    ptrs = (C.c_void_p * 6)(*[t.data_ptr() for t in slabs])
    sp = np.ascontiguousarray(specs, np.float32)
    L = fg.lib()
    for n in range(STEPS):
        f = st.fields(n, True)
        if static:
            fg.check(L.fdtd_step_static(C.byref(raw), fg.fptr(sp), len(sp), fg.SCHEME_CORRECTED, C.byref(f), ptrs, n,
                                        None), "fdtd_step_static")
        else:
            fg.check(L.fdtd_step(plan.handle, C.byref(f), n, None), "fdtd_step")
    torch.cuda.synchronize()
    if plan:
        plan.close()
    return st.latest(STEPS, True)


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("dims,shift", [((33, 9, 6), 0), ((17, 10, 5), 0), ((32, 9, 6), 1), ((32, 9, 6), 0)])
def test_bytes_beyond_the_table_take_its_last_class(cuda, dims, shift, static):
    codes, beyond, specs, rp, raw = _case(dims)
    want = _run(cuda, dims, raw, codes, specs, rp, static, shift)
    got = _run(cuda, dims, raw, beyond, specs, rp, static, shift)
    assert np.any(want["ez"])
    for name in want:
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name


def test_two_pass_step_has_a_zero_row_for_them(cuda):
    dims = (33, 9, 6)
    codes, beyond, specs, rp, raw = _case(dims)
    nx, ny, nz = dims
    plan = fg.Plan(Params(raw), specs, scheme=fg.SCHEME_CORRECTED, rp=rp)
    st = NativeState(cuda, (nz, ny, nx), beyond)
    gen = cuda.Generator(device="cuda")
    gen.manual_seed(1)
    for v in (*st.e[0], *st.e[1]):
        v.copy_(cuda.randn(v.shape, generator=gen, device="cuda"))
    f = st.fields(0, False)
    fg.check(fg.lib().fdtd_step_de(plan.handle, C.byref(f), 0, None), "fdtd_step_de")
    cuda.cuda.synchronize()
    plan.close()
    e = st.latest(1, False)
    inner = np.zeros(beyond.shape, bool)
    inner[2:-2, 2:-2, 2:-2] = True  # clear of the Mur faces
    for name in ("ex", "ey", "ez"):
        assert np.all(e[name][inner & (beyond >= NCLS)] == 0.0), name
        assert np.all(e[name][inner & (beyond < NCLS)] != 0.0), name
