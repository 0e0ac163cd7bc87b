"""Snapshots taken beside running steps, dense rows (copied from the state) and
padded ones (packed into one staging area first, which the next snapshot packs
over): every snapshot of a run in one call holds the fields after its step, bit
for bit, at short and long intervals and with planes of the grid only."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [fg.KERNEL_SINGLE_PASS, fg.KERNEL_TWO_PASS, fg.KERNEL_COMPACT_R16])
@pytest.mark.parametrize("dims,z0,nplanes", [((121, 90, 60), 0, 0), ((121, 90, 60), 7, 3), ((128, 90, 60), 0, 0)])
@pytest.mark.parametrize("every", [1, 3])
def test_snapshots_of_a_running_solve(cuda, dims, z0, nplanes, every, kernel):
    steps, fields = 13, ("hx", "ey", "ez")
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=6, ncls=3, nsrc=3)
    p = Params(make_params(dims, consts, sources, jz))
    got = {}
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.set_snapshots(every, fields=fields, z0=z0, nplanes=nplanes,
                        callback=lambda step, name, a: got.__setitem__((step, name), a))
        s.run(steps)
        s.flush_snapshots()
    planes = slice(z0, z0 + (nplanes or dims[2]))
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        for step in range(steps):
            s.run(1)
            for name in fields if step % every == 0 else ():
                want = s.field(name)[planes]
                assert got.pop((step, name)).tobytes() == want.tobytes(), (step, name)
    assert not got
