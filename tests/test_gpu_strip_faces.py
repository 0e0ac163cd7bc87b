"""The x faces in the strip kernel's tiles, updated by its moving warp: grids
whose near and far face share a tile (rows of 17 to 32 cells), whose far face
lies in a tile's second, last or first column (the last is the Mur kernel's),
tile rows beyond the grid, the smallest y and z, chunks that begin on either
side of the z faces; in every strip shape, against the z-marching kernel (which
applies the same rounded operations in its cell threads) bit for bit, in both
schemes (whose far ey face differs) and both storage forms."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [0, 1, 2, 3])
@pytest.mark.parametrize("kernel", [fg.KERNEL_COMPACT, fg.KERNEL_COMPACT_R16])
@pytest.mark.parametrize("scheme", [fg.SCHEME_REFERENCE, fg.SCHEME_CORRECTED])
@pytest.mark.parametrize("dims", [(17, 9, 5), (31, 3, 9), (32, 16, 3), (33, 17, 6), (34, 7, 41), (63, 10, 12),
                                  (66, 18, 4)])
def test_faces_equal_the_z_marching_kernel(cuda, monkeypatch, dims, scheme, kernel, shape):
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=sum(dims), ncls=4, nsrc=2)
    sources = [*sources, (1, 1, 1), (dims[0] - 2, dims[1] - 2, dims[2] - 2)]  # so that the faces carry a field
    p = Params(make_params(dims, consts, sources, jz))
    out = {}
    for step in ("strip", "zmarch"):
        if step == "zmarch":
            monkeypatch.setenv("FDTD_COMPACT_STEP", "zmarch")
        else:
            monkeypatch.setenv("FDTD_STRIP_SHAPE", str(shape))
        with fg.Solver(p, codes, specs, scheme=scheme, kernel=kernel, nclasses=len(specs)) as s:
            s.run(16)
            out[step] = s.fields()
    for side in (0, -1):
        assert np.count_nonzero(out["strip"]["ey"][:, :, side]) and np.count_nonzero(out["strip"]["ez"][:, :, side])
    for name, want in out["zmarch"].items():
        assert np.array_equal(out["strip"][name].view(np.uint32), want.view(np.uint32)), name
