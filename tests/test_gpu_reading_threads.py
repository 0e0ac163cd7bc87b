"""Several threads reading one solver at once.  Reads into pageable memory of
grids with padded rows go through the solver's staging area, which the threads
share: each must get its own field, bit for bit."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(150, 120, 260), (33, 20, 11)])  # more than a staging area, and less
def test_threads_read_their_own_fields(cuda, dims):
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=4, ncls=3, nsrc=3)
    p = Params(make_params(dims, consts, sources, jz))
    names = ["ex", "ey", "ez", "hx", "hy", "hz"]
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED) as s:
        s.run(60)
        want = {n: s.field(n) for n in names}
        assert len({want[n].tobytes() for n in names}) == len(names)
        wrong, start = [], threading.Barrier(len(names))

        def read(name):
            out = np.zeros(p.shape, np.float32)
            start.wait()
            for _ in range(12):
                out.fill(0.0)
                s.field(name, out=out)
                if not np.array_equal(out.view(np.uint32), want[name].view(np.uint32)):
                    wrong.append(name)

        threads = [threading.Thread(target=read, args=(n,)) for n in names]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong
