"""A cell's update does not depend on where z chunks meet, with both sides of
each comparison sure to run in chunks of other lengths: long ones by a grid or
a batch of many blocks (beyond eight waves the longest chunk is taken), short
ones by a small grid, and set ones through FDTD_STRIP_ZCHUNK."""
from __future__ import annotations

import os

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu

FORMS = [fg.KERNEL_SINGLE_PASS, fg.KERNEL_COMPACT, fg.KERNEL_COMPACT_R16]


def _equal(got, want):
    assert any(np.any(v) for v in want.values())
    for name in want:
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name


@pytest.mark.parametrize("kernel", FORMS)
def test_sources_on_the_borders_of_long_chunks(cuda, kernel):
    """1664 column tiles of 130 planes, cut at planes 44 and 88 (D form) or 33, 66
    and 99: sources on both sides of those, each in a column of its own.  In six
    steps each one's field stays within seven cells, and equals that of the same
    source alone on a small grid."""
    dims, small, steps, reach = (1024, 416, 130), (40, 40, 40), 6, 8
    consts = random_case(8, 8, 8, seed=1, ncls=2, nsrc=0)[4]
    jz = np.linspace(1.0, 2.0, 16).astype(np.float32)
    specs = np.array([[0.0, 1.0, 1.0, 0.0], [0.5, 30.0, 5.0, 1e-11]], np.float32)
    planes = [32, 33, 34, 43, 44, 45, 65, 66, 67, 87, 88, 98, 99]
    at = [(25 + 71 * k, 40 + 26 * k, z) for k, z in enumerate(planes)]
    p = Params(make_params(small, consts, [(20, 20, 20)], jz))
    with fg.Solver(p, np.ones(small[::-1], np.uint8), specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(steps)
        near = slice(20 - reach, 21 + reach)
        want = {n: v[near, near, near] for n, v in s.fields().items()}
        assert all(np.count_nonzero(v) == np.count_nonzero(want[n]) for n, v in s.fields().items())
    p = Params(make_params(dims, consts, at, jz))
    with fg.Solver(p, np.ones(dims[::-1], np.uint8), specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(steps)
        for name, w in want.items():
            field = s.field(name)
            assert np.count_nonzero(field) == len(at) * np.count_nonzero(w), name
            for x, y, z in at:
                box = field[z - reach:z + reach + 1, y - reach:y + reach + 1, x - reach:x + reach + 1]
                assert np.array_equal(box.view(np.uint32), np.ascontiguousarray(w).view(np.uint32)), (name, x, y, z)


@pytest.mark.parametrize("kernel", FORMS)
@pytest.mark.parametrize("dims", [(64, 16, 65), (48, 30, 129), (96, 40, 67)])
def test_a_small_solve_beside_a_large_one(cuda, dims, kernel):
    """Alone the small grid runs in chunks of a few planes; in a batch with 5120
    column-tile chunks of a large one it runs in the form's longest."""
    steps = 14
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=sum(dims), ncls=4, nsrc=3)
    codes[:, : dims[1] // 2, :] = 0
    p = Params(make_params(dims, consts, sources, jz))
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(steps)
        want = s.fields()
    large = (640, 512, 200)
    q = Params(make_params(large, consts, [(300, 200, 100)], jz))
    b = fg.Batch(0, kernel)
    b.add(q, np.zeros(large[::-1], np.uint8), np.array([[0, 1, 1, 0]], np.float32), steps, scheme=fg.SCHEME_CORRECTED)
    sid = b.add(p, codes, specs, steps, scheme=fg.SCHEME_CORRECTED)
    b.run(steps)
    got = b.fields(sid)
    b.close()
    _equal(got, want)


@pytest.mark.parametrize("kernel", FORMS[1:])
def test_set_chunk_lengths(cuda, kernel, monkeypatch):
    dims, steps = (70, 26, 150), 20
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=5, ncls=3, nsrc=4)
    codes[:, :13, :] = 0  # memoryless tile-planes too
    p = Params(make_params(dims, consts, sources, jz))
    runs = {}
    for limit in (None, 2, 7, 24, 50, 64):
        if limit is None:
            monkeypatch.delenv("FDTD_STRIP_ZCHUNK", raising=False)
        else:
            monkeypatch.setenv("FDTD_STRIP_ZCHUNK", str(limit))
        with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
            s.run(steps)
            runs[limit] = s.fields()
    assert "FDTD_STRIP_ZCHUNK" in os.environ
    for limit, got in runs.items():
        _equal(got, runs[2])
