"""Dense rows read into page-locked memory at and around the length from which
the kernel writes them instead of the copy engine: the same bytes as a read into
pageable memory, at any offset from a 16-byte boundary."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params

pytestmark = pytest.mark.gpu

LONG_FLOATS = 16 << 20


@pytest.mark.parametrize("dims", [(256, 256, 255), (256, 256, 256), (256, 256, 257)])
def test_both_sides_of_the_limit(cuda, dims):
    n = int(np.prod(dims))
    assert (n >= LONG_FLOATS) == (dims[2] >= 256)
    consts = dict(dt=1.9e-12, dx=1e-3, dy=1e-3, dz=1e-3, mu0=1.2566e-6, eps0=8.8542e-12)
    p = Params(make_params(dims, consts, [(100, 120, 6), (90, 80, 249)], np.ones(16, np.float32)))
    codes = np.zeros(dims[::-1], np.uint8)
    raw = cuda.zeros(n + 4, pin_memory=True).numpy()
    with fg.Solver(p, codes, np.array([[0, 1, 1, 0]], np.float32)) as s:
        s.run(12)
        want = s.field("ez")
        assert np.any(want[:10]) and np.any(want[-10:])
        for skew in (0, 1):
            out = raw[skew:skew + n].reshape(codes.shape)
            out[:] = -1.0
            s.field("ez", out=out)
            assert out.tobytes() == want.tobytes(), skew
