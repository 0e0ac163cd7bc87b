"""Memoryless tile-planes of a solver, found on the device: the share it
reports equals a count on the host for volumes with partial tiles in x and y,
a partial last z chunk, padded rows, every tile height, and none or all cells
without relaxation; and skipping R there changes no bit against the
z-marching kernel, which skips nothing."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


def _share(codes, memless, rows):
    nz, ny, nx = codes.shape
    cells = 0
    for y in range(0, ny, rows):
        for x in range(0, nx, 32):
            tile = memless[codes[:, y:y + rows, x:x + 32]]
            cells += int(tile.all(axis=(1, 2)).sum()) * tile.shape[1] * tile.shape[2]
    return cells / codes.size


@pytest.mark.parametrize("shape", [0, 3])
@pytest.mark.parametrize("kernel", [fg.KERNEL_COMPACT, fg.KERNEL_COMPACT_R16])
@pytest.mark.parametrize("dims,fill", [((48, 17, 5), 0.5), ((70, 33, 41), 0.02), ((33, 9, 90), 0.3), ((96, 24, 7), 0.0),
                                       ((64, 16, 8), 1.0)])
def test_share_and_fields(cuda, monkeypatch, dims, fill, kernel, shape):
    nx, ny, nz = dims
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=nx + nz, ncls=4, nsrc=2)
    specs[:, 3] = np.where(np.arange(len(specs)) % 2 == 0, 0.0, np.maximum(specs[:, 3], 5e-12))
    rng = np.random.default_rng(nz)
    codes = np.zeros((nz, ny, nx), np.uint8)
    codes[rng.random(codes.shape) < fill * 0.02] = 1
    if fill == 1.0:
        codes[:] = 1
    codes[nz // 2, : ny // 2] = 2
    p = Params(make_params(dims, consts, sources, jz))
    monkeypatch.setenv("FDTD_STRIP_SHAPE", str(shape))
    out = []
    for step in ("strip", "zmarch"):
        monkeypatch.setenv("FDTD_COMPACT_STEP", step)
        with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
            assert s.memless_fraction == _share(codes, specs[:, 3] == 0.0, 16 if shape == 3 else 8)
            s.run(20)
            out.append(s.fields())
    for name, want in out[1].items():
        assert np.array_equal(out[0][name].view(np.uint32), want.view(np.uint32)), name
