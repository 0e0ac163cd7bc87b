"""The compat launchers at the edges of their launch shapes: planes below, at
and just over the H and D kernels' planes per thread, rows and columns around
one 64 x 2 tile, more rows than a grid has blocks in y, face rows around the
Mur kernel's rows per thread, and calls queued back to back on one stream (each
launch may be placed before the previous one has finished, and must still read
what it wrote).  Against the FP32 oracle (the
reference kernels' own arithmetic), 24 rotated steps, at the parity bar of
every field."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import fdtd_gb300 as fg
from oracle import pyoracle as po

from .gpu_util import dev, make_params, ptr, zeros
from .helpers import assert_fields_close, class_media, random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 3, 3), (31, 8, 4), (32, 9, 5), (33, 7, 6), (34, 16, 8), (65, 17, 9),
                                  (130, 5, 13), (5, 131, 10), (63, 3, 5), (64, 4, 4), (3, 131074, 3)])
def test_back_to_back_steps_match_the_oracle(cuda, dims):
    torch, (nx, ny, nz), steps = cuda, dims, 24
    codes, specs, rp, sources, consts, jz = random_case(*dims, seed=sum(dims), ncls=3, nsrc=2)
    media = class_media(codes, specs, rp)
    raw = make_params(dims, consts, sources, jz)
    L = fg.lib()
    fg.check(L.fdtd_copy_symbols(C.byref(raw)), "fdtd_copy_symbols")
    shape = (nz, ny, nx)
    h = [zeros(torch, shape) for _ in range(3)]
    e = [[zeros(torch, shape) for _ in range(3)] for _ in range(3)]
    d = [[zeros(torch, shape) for _ in range(3)] for _ in range(3)]
    mats = [dev(torch, specs[codes, k].astype(np.float32)) for k in (0, 2, 1, 3)]  # sigma, eps_inf, eps_s, tau
    slabs = [dev(torch, r) for r in rp]
    p = lambda ts: [ptr(t) for t in ts]  # noqa: E731
    for n in range(steps):
        t, n0, n1 = n % 3, (n + 2) % 3, (n + 1) % 3
        fg.check(L.fdtd_update_h(*p(h), *p(e[n0]), None))
        fg.check(L.fdtd_update_d(*p(d[t]), *p(d[n0]), *p(h), None))
        fg.check(L.fdtd_update_sources(ptr(d[t][2]), ptr(d[n0][2]), ptr(h[0]), ptr(h[1]), n - n % 3, None))
        fg.check(L.fdtd_update_e(*p(e[t]), *p(e[n0]), *p(e[n1]), *p(d[t]), *p(d[n0]), *p(d[n1]), *p(mats), None))
        fg.check(L.fdtd_update_mur(*p(e[t]), *p(e[n0]), *p(slabs), None))
    torch.cuda.synchronize()
    k = (steps - 1) % 3
    got = {f"{f}{c}": v[i].cpu().numpy() for f, v in (("h", h), ("e", e[k]), ("d", d[k])) for i, c in enumerate("xyz")}
    st = po.State(*dims, np.float32)
    po.run(po.make_cfg(dims, jz, sources=sources, consts=consts), media, st, 0, steps)
    want = st.latest(steps)
    assert all(np.all(np.isfinite(want[v])) for v in want)
    assert_fields_close(got, want, names=list(got))
