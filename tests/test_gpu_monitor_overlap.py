"""Monitors beside overlapped steps: inside a step graph the next step's
kernel starts while the monitor kernel of this one still runs.  On a grid with
blocks clear of the faces (those start early) the probe series, the DFT sums
and the fields of a run in whole graphs must equal, bit for bit, a run that
waits after every step."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [fg.KERNEL_SINGLE_PASS, fg.KERNEL_TWO_PASS, fg.KERNEL_COMPACT,
                                    fg.KERNEL_COMPACT_R16])
@pytest.mark.parametrize("stride", [0, 1, 3])
def test_overlapped_monitors_equal_serial_ones(cuda, kernel, stride):
    dims, steps = (151, 50, 90), 48
    codes, specs, _, _, consts, jz = random_case(*dims, seed=31, ncls=4, nsrc=0)
    sources = [(75, 25, 45), (3, 2, 1), (100, 30, 50)]
    p = Params(make_params(dims, consts, sources, jz))
    probes = [(75, 25, 45), (0, 0, 0), (150, 49, 89), (40, 20, 30), (76, 25, 45)]
    runs = []
    for serial in (False, True):
        with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
            s.set_probes(probes, capacity=steps)
            if stride:
                s.set_dft(1.1e9, stride=stride, z0=5, nplanes=70)
            if serial:
                for _ in range(steps):
                    s.run(1)
                    s.synchronize()
            else:
                s.run(steps)
            out = dict(s.fields(), probes=s.probes())
            if stride:
                for c in range(3):
                    out[f"dft{c}"] = s.dft(c).view(np.float64)
            runs.append(out)
    assert np.any(runs[1]["probes"][:, 0])
    for name, want in runs[1].items():
        got = runs[0][name]
        bits = np.uint64 if want.dtype == np.float64 else np.uint32
        assert np.array_equal(got.view(bits), want.view(bits)), name
