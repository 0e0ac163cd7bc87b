"""fdtd_solver_profile names and times the kernels that a step of the solve
runs: a D-form grid whose rows TMA cannot address takes the two-pass kernels.
Its steps are real ones."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,kernel,names", [
    ((32, 9, 6), fg.KERNEL_SINGLE_PASS, {"fused_step", "mur"}),
    ((61, 9, 6), fg.KERNEL_SINGLE_PASS, {"fused_step", "mur"}),  # padded rows
    ((10, 9, 6), fg.KERNEL_SINGLE_PASS, {"h", "de", "mur"}),
    ((33, 9, 6), fg.KERNEL_SINGLE_PASS, {"h", "de", "mur"}),
    ((33, 9, 6), fg.KERNEL_TWO_PASS, {"h", "de", "mur"}),
    ((33, 9, 6), fg.KERNEL_COMPACT, {"compact_step", "mur"}),
])
def test_the_kernels_of_a_step(cuda, dims, kernel, names):
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=8, ncls=3, nsrc=2)
    sources = sources + [(dims[0] - 1, dims[1] - 1, dims[2] - 1)]
    p = Params(make_params(dims, consts, sources, jz))
    fields = []
    for profiled in (True, False):
        with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
            s.run(3)
            if profiled:
                ms = s.profile(4)
                assert set(ms) == names and all(v > 0.0 for v in ms.values())
            else:
                s.run(4)
            s.run(3)
            fields.append(s.fields())
    for name, want in fields[1].items():
        assert np.array_equal(fields[0][name].view(np.uint32), want.view(np.uint32)), name
