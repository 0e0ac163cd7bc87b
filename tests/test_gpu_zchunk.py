"""z chunks of a single solve's launch (balanced_zchunk): small and middle grids
run in chunks chosen by whole waves of CTAs, down to two planes.  A cell's
update does not depend on where chunks meet, so every field must equal, bit
for bit, the same solve in a batch of one (which runs the form's default
chunks), on grids whose plane counts leave full, short and single-plane last
chunks, with sources and memoryless tile-planes in them."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu

# planes: below, at and just over small multiples of 2 and 3; one grid of several waves
DIMS = [(16, 8, 3), (32, 8, 4), (64, 16, 5), (64, 64, 64), (48, 30, 65), (96, 80, 67), (144, 120, 129)]


@pytest.mark.parametrize("kernel", [fg.KERNEL_SINGLE_PASS, fg.KERNEL_COMPACT, fg.KERNEL_COMPACT_R16])
@pytest.mark.parametrize("dims", DIMS)
def test_chunk_length_does_not_change_a_bit(cuda, dims, kernel):
    nx, ny, nz = dims
    steps = 18
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=sum(dims), ncls=4, nsrc=2)
    codes[:, : ny // 2, :] = 0
    sources = sources + [(1, 1, 0), (nx - 1, ny - 1, nz - 1), (nx // 2, ny // 2, min(2, nz - 1))]
    p = Params(make_params(dims, consts, sources, jz))
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(steps)
        got = s.fields()
    b = fg.Batch(0, kernel)
    sid = b.add(p, codes, specs, steps, scheme=fg.SCHEME_CORRECTED)
    b.run(steps)
    want = b.fields(sid)
    b.close()
    assert sorted(got) == sorted(want)
    assert any(np.any(v) for v in want.values())
    for name in want:
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name
