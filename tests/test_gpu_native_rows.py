"""fdtd_step and fdtd_step_static on a caller's own buffers that TMA cannot
address -- rows that are not a multiple of 16 cells, bases off 16 bytes -- run
the two-pass kernels; the same steps on addressable buffers run the
single-pass kernel.  Both against the FP64 oracle (corrected scheme) and each
other, with non-uniform Mur slabs, over grids with partial tiles and the far x
face at every place in a tile."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import fdtd_gb300 as fg
from oracle import pyoracle as po

from .gpu_util import NativeState, Params, make_params
from .helpers import REL_L2_TOL, class_media, random_case, rel_l2

pytestmark = pytest.mark.gpu


def _shift(torch, st, floats):
    """Moves every array of the state to a base `floats` elements off 16 bytes."""
    for slots in (st.h, st.e, st.d):
        for slot in slots:
            for k in range(3):
                v = slot[k]
                big = torch.zeros(v.numel() + 4, dtype=v.dtype, device=v.device)
                slot[k] = big[floats:floats + v.numel()].view(v.shape)


@pytest.mark.parametrize("dims,shift", [((17, 9, 6), 0), ((31, 8, 5), 0), ((33, 10, 9), 0), ((34, 7, 4), 0),
                                        ((61, 33, 12), 0), ((48, 9, 7), 1), ((32, 16, 5), 3), ((48, 9, 7), 0)])
@pytest.mark.parametrize("static", [False, True])
def test_callers_rows_match_the_oracle(cuda, dims, shift, static):
    torch, (nx, ny, nz), steps = cuda, dims, 18
    codes, specs, rp, sources, consts, jz = random_case(*dims, seed=sum(dims), ncls=3, nsrc=2)
    raw = make_params(dims, consts, sources, jz)
    plan = fg.Plan(Params(raw), specs, scheme=fg.SCHEME_CORRECTED, rp=rp)
    st = NativeState(torch, (nz, ny, nx), codes)
    if shift:
        _shift(torch, st, shift)
    L = fg.lib()
    slabs = [torch.from_numpy(np.ascontiguousarray(r)).cuda() for r in rp]
    ptrs = (C.c_void_p * 6)(*[t.data_ptr() for t in slabs])
    sp = np.ascontiguousarray(specs, np.float32)
    for n in range(steps):
        f = st.fields(n, True)
        if static:
            fg.check(L.fdtd_step_static(C.byref(raw), fg.fptr(sp), len(sp), fg.SCHEME_CORRECTED, C.byref(f), ptrs, n,
                                        None), "fdtd_step_static")
        else:
            fg.check(L.fdtd_step(plan.handle, C.byref(f), n, None), "fdtd_step")
    torch.cuda.synchronize()
    got = st.latest(steps, True)
    plan.close()
    media = class_media(codes, specs, rp)
    cfg = po.make_cfg(dims, jz, sources=sources, consts=consts, corrected=True)
    ref, f32 = po.State(*dims, np.float64), po.State(*dims, np.float32)
    po.run(cfg, media, ref, 0, steps)
    po.run(cfg, media, f32, 0, steps)
    want, single = ref.latest(steps), f32.latest(steps)
    for name in got:
        # the parity bar, or twice the reference's own single-precision error where that is larger
        bound = max(REL_L2_TOL, 2.0 * rel_l2(single[name], want[name]))
        assert rel_l2(got[name], want[name]) <= bound, (name, rel_l2(got[name], want[name]), bound)


def test_sources_on_upper_faces_read_h_where_it_is_never_updated(cuda):
    # H cells outside the update ranges hold their value in h_in only; the other buffer holds NaN.  The
    # single-pass kernel (addressable bases) and the two-pass kernels (bases off 16 bytes) must agree.
    torch, dims = cuda, (32, 9, 6)
    nx, ny, nz = dims
    codes, specs, rp, _, consts, jz = random_case(*dims, seed=5, ncls=2, nsrc=1)
    sources = [(nx - 1, ny - 1, nz - 1), (nx - 1, 3, 2), (7, ny - 1, 2), (9, 4, nz - 1), (5, 5, 3), (1, 1, 0)]
    raw = make_params(dims, consts, sources, jz + 1.0)
    plan = fg.Plan(Params(raw), specs, scheme=fg.SCHEME_CORRECTED, rp=rp)
    out = []
    for shift in (0, 1):
        st = NativeState(torch, (nz, ny, nx), codes)
        if shift:
            _shift(torch, st, shift)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(3)
        for k in range(3):
            st.h[0][k].copy_(torch.randn(st.h[0][k].shape, generator=gen, device="cuda"))
            st.h[1][k].fill_(float("nan"))
        f = st.fields(0, True)
        fg.check(fg.lib().fdtd_step(plan.handle, C.byref(f), 0, None), "fdtd_step")
        torch.cuda.synchronize()
        out.append(st.latest(1, True))
    plan.close()
    for name in ("dx", "dy", "dz", "ex", "ey", "ez"):
        assert np.all(np.isfinite(out[0][name])) and np.all(np.isfinite(out[1][name])), name
        assert rel_l2(out[1][name], out[0][name]) <= 1e-6, name
