"""Checkpoints of solves with padded rows: the file holds the dense blocks of
the fields, in the order H, E^n, E^{n-1} and the form's history, whatever the
rows' padding and however long the volume, and gives the state back."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [fg.KERNEL_SINGLE_PASS, fg.KERNEL_TWO_PASS, fg.KERNEL_COMPACT,
                                    fg.KERNEL_COMPACT_R16])
@pytest.mark.parametrize("dims", [(17, 9, 6), (131, 150, 230)])
def test_file_holds_dense_rows_and_restores(cuda, tmp_path, dims, kernel):
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=3, ncls=3, nsrc=3)
    p = Params(make_params(dims, consts, sources, jz))
    path = tmp_path / "ck.bin"
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(9)
        fields = s.fields()
        s.checkpoint(path)
        s.run(4)
        want = s.fields()
    n = codes.size
    data = path.read_bytes()
    d_form = kernel in (fg.KERNEL_SINGLE_PASS, fg.KERNEL_TWO_PASS)
    history = 24 if d_form else 12 if kernel == fg.KERNEL_COMPACT else 6
    header = len(data) - n * (36 + history)
    if kernel != fg.KERNEL_COMPACT_R16:  # that form's scale words follow
        assert 0 < header < 256
    blocks = ["hx", "hy", "hz", "ex", "ey", "ez"] + [None] * 3 + (["dx", "dy", "dz"] if d_form else [])
    at = header if kernel != fg.KERNEL_COMPACT_R16 else data.find(fields["hx"].tobytes())
    assert at > 0
    for k, name in enumerate(blocks):
        if name:
            assert data[at + 4 * n * k:at + 4 * n * (k + 1)] == fields[name].tobytes(), name
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(2)
        s.restore(path)
        s.run(4)
        got = s.fields()
    for name in want:
        assert got[name].tobytes() == want[name].tobytes(), name
