"""Solves that join and leave a running batch: the batch's descriptors, tensor
maps among them, change in place at every turn.  Each solve's fields must equal,
bit for bit, the same solve run alone."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu

DIMS = [(40, 20, 12), (17, 33, 9), (70, 9, 21), (33, 16, 30), (96, 24, 8)]


@pytest.mark.parametrize("kernel", [fg.KERNEL_SINGLE_PASS, fg.KERNEL_COMPACT, fg.KERNEL_COMPACT_R16])
def test_descriptors_that_change_in_place(cuda, kernel):
    b = fg.Batch(0, kernel)
    live = []
    for turn in range(15):
        dims = DIMS[turn % len(DIMS)]
        codes, specs, _, sources, consts, jz = random_case(*dims, seed=200 + turn, ncls=3, nsrc=2)
        p = Params(make_params(dims, consts, sources, jz))
        live.append([b.add(p, codes, specs, 1 << 20, scheme=fg.SCHEME_CORRECTED), p, codes, specs, 0])
        b.run(3)
        for v in live:
            v[4] += 3
        if len(live) < 4:
            continue
        sid, p, codes, specs, steps = live.pop(0)  # every later solve moves up one descriptor
        got = b.fields(sid)
        b.remove(sid)
        with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
            s.run(steps)
            want = s.fields()
        assert np.any(want["ez"])
        for name in want:
            assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), (turn, name)
    b.close()
