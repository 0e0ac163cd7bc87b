"""Every bounded wait that gives up is reported, whichever warp waits.  The
hooks make a wait of one CTA give up without a GPU fault: its loads never come
(fdtd_solver_test_stall), or the warp that stores the finished tiles gives up
while the cell warps finish their last planes (fdtd_solver_test_stall_store).
FDTD_ERR_DEVICE_TIMEOUT comes once, soon; the context stays usable, and a
checkpoint restored gives the bits of an undisturbed run."""
from __future__ import annotations

import time

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu


def _problem(dims=(70, 20, 30)):
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=9, ncls=3, nsrc=2)
    return Params(make_params(dims, consts, sources, jz)), codes, specs


@pytest.mark.parametrize("kernel,hook", [(fg.KERNEL_COMPACT, "test_stall_store"), (fg.KERNEL_COMPACT_R16, "test_stall_store"),
                                         (fg.KERNEL_COMPACT_R16, "test_stall")])
def test_solver_reports_a_wait_that_gave_up(cuda, tmp_path, kernel, hook):
    p, codes, specs = _problem()
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(6)
        s.checkpoint(tmp_path / "ck.bin")
        getattr(s, hook)()
        t0 = time.perf_counter()
        s.run(1)
        with pytest.raises(fg.FdtdError) as e:
            s.synchronize()
        assert e.value.status == fg.FDTD_ERR_DEVICE_TIMEOUT
        assert time.perf_counter() - t0 < 5.0
        s.run(2)
        s.synchronize()  # reported once; later steps run
        s.restore(tmp_path / "ck.bin")
        s.run(10)
        got = s.fields()
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.run(16)
        want = s.fields()
    for name in want:
        assert np.array_equal(got[name].view(np.uint32), want[name].view(np.uint32)), name


def test_batch_reports_a_wait_that_gave_up(cuda):
    b = fg.Batch(0, fg.KERNEL_SINGLE_PASS)
    cases = [_problem(), _problem((33, 40, 12)), _problem((50, 9, 40))]
    ids = [b.add(p, codes, specs, 1 << 20, scheme=fg.SCHEME_CORRECTED) for p, codes, specs in cases]
    b.run(6)
    b.synchronize()
    b.test_stall(ids[1])
    t0 = time.perf_counter()
    b.run(1)
    with pytest.raises(fg.FdtdError) as e:
        b.synchronize()
    assert e.value.status == fg.FDTD_ERR_DEVICE_TIMEOUT
    assert time.perf_counter() - t0 < 5.0
    b.run(3)
    b.synchronize()  # reported once; later steps run
    # the other solves are as if nothing had happened
    for sid, (p, codes, specs) in ((ids[0], cases[0]), (ids[2], cases[2])):
        got = b.fields(sid)
        with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED) as s:
            s.run(10)
            for name, want in s.fields().items():
                assert np.array_equal(got[name].view(np.uint32), want.view(np.uint32)), name
    b.close()


def test_forms_without_a_hook_refuse_it(cuda):
    p, codes, specs = _problem()
    for kernel in (fg.KERNEL_SINGLE_PASS, fg.KERNEL_TWO_PASS):
        with fg.Solver(p, codes, specs, kernel=kernel) as s:
            with pytest.raises(fg.FdtdError):
                s.test_stall_store()
    b = fg.Batch(0, fg.KERNEL_COMPACT)
    sid = b.add(p, codes, specs, 10)
    with pytest.raises(fg.FdtdError):
        b.test_stall(sid)
    b.close()
