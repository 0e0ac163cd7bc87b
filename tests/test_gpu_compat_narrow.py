"""The compat launchers on grids narrower than a 64-wide tile, at and around
the widths where the tile changes (8, 16 and 32 cells), with rows just below, at
and above a tile's: as test_gpu_compat_shapes."""
from __future__ import annotations

import pytest

from .test_gpu_compat_shapes import test_back_to_back_steps_match_the_oracle as _matches_the_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(7, 15, 5), (8, 16, 6), (9, 17, 9), (15, 9, 4), (16, 8, 7), (17, 7, 5), (33, 5, 6)])
def test_narrow_grids(cuda, dims):
    _matches_the_oracle(cuda, dims)
