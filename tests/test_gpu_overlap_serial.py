"""Overlapped steps against truly serial ones.  Inside a step graph the next
step's kernel starts while the Mur kernel of this one still runs, also where
monitors are installed; a run that waits on the host after every step overlaps
nothing.  On grids with blocks clear of the faces, and sources near faces and
inside, both must give the same bits, without monitors, in every form."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [fg.KERNEL_SINGLE_PASS, fg.KERNEL_TWO_PASS, fg.KERNEL_COMPACT,
                                    fg.KERNEL_COMPACT_R16])
@pytest.mark.parametrize("dims", [(160, 48, 140), (151, 50, 90)])
def test_overlapped_steps_equal_steps_with_a_wait_after_each(cuda, dims, kernel):
    steps = 90
    codes, specs, _, _, consts, jz = random_case(*dims, seed=21, ncls=4, nsrc=0)
    nx, ny, nz = dims
    sources = [(nx // 2, ny // 2, nz // 2), (3, 2, 1), (nx - 2, ny - 2, nz - 2), (100, 30, 50)]
    p = Params(make_params(dims, consts, sources, jz))
    runs = []
    for serial in (False, True):
        with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
            for chunk in [1] * steps if serial else (7, 40, 43):
                s.run(chunk)
                if serial:
                    s.synchronize()
            runs.append(s.fields())
    assert np.any(runs[1]["ez"])
    for name, want in runs[1].items():
        assert np.array_equal(runs[0][name].view(np.uint32), want.view(np.uint32)), name
