"""Solves whose rows are padded on the device (nx not a multiple of 16): every
way a volume leaves or enters the solver sees the dense grid -- reads into
pageable and page-locked memory (a kernel writes the latter), reads longer
than the staging area, snapshots, probes, the running DFT and its peak SAR
cell, checkpoints -- all checked against each other bit for bit, and the
fields against a batch of one."""
from __future__ import annotations

import numpy as np
import pytest

import fdtd_gb300 as fg

from .gpu_util import Params, make_params
from .helpers import random_case

pytestmark = pytest.mark.gpu

KERNELS = [fg.KERNEL_SINGLE_PASS, fg.KERNEL_TWO_PASS, fg.KERNEL_COMPACT, fg.KERNEL_COMPACT_R16]


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32 if a.dtype.itemsize == 4 else np.uint64)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("dims", [(17, 9, 6), (15, 12, 7), (33, 10, 5), (47, 21, 19)])
def test_every_exit_sees_the_dense_grid(cuda, tmp_path, dims, kernel):
    nx, ny, nz = dims
    steps, stride, freq = 12, 3, 1.0e9
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=nx + ny, ncls=4, nsrc=3)
    p = Params(make_params(dims, consts, sources, jz))
    probes = [(0, 0, 0), (nx - 1, ny - 1, nz - 1), (nx - 1, 0, nz // 2), sources[0]]
    shots = {}
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.set_probes(probes, capacity=steps)
        s.set_dft(freq, stride=stride, z0=1, nplanes=nz - 2)
        s.set_snapshots(1, fields=("hx", "ez"), z0=1, nplanes=2,
                        callback=lambda step, name, a: shots.__setitem__((step, name), a))
        acc = np.zeros((3, nz - 2, ny, nx), np.complex128)
        series = []
        for n in range(steps):
            s.run(1)
            e = [s.field(k) for k in ("ex", "ey", "ez")]
            series.append([[v[z, y, x] for v in e] for x, y, z in probes])
            s.flush_snapshots()
            assert np.array_equal(_bits(shots[n, "ez"]), _bits(e[2][1:3]))
            assert np.array_equal(_bits(shots[n, "hx"]), _bits(s.field("hx")[1:3]))
            if (n + 1) % stride == 0:
                t = (n + 1) * p.dt  # the single-precision time step the library is given
                ph = np.exp(-2j * np.pi * freq * t) * stride * p.dt
                for c in range(3):
                    acc[c] += e[c][1:nz - 1].astype(np.float64) * ph
        assert np.array_equal(_bits(s.probes()), _bits(np.array(series, np.float32)))
        for c in range(3):
            assert np.allclose(s.dft(c), acc[c], rtol=1e-10, atol=1e-12 * np.abs(acc[c]).max())
        peak, cell = s.peak_sar()
        sar = specs[codes[1:nz - 1], 0] * (np.abs(acc) ** 2).sum(0) / 2000.0
        assert abs(peak - sar.max()) <= 1e-6 * sar.max()  # sigma and 1/(2 rho) are single precision
        z, y, x = np.unravel_index(cell, (nz, ny, nx))
        assert sar[z - 1, y, x] >= sar.max() * (1 - 1e-6)
        want = s.fields()
        pinned = fg.PinnedBuffer(codes.size)
        for name, v in want.items():
            assert np.array_equal(_bits(s.field(name, out=pinned.view(codes.shape))), _bits(v)), name
        s.checkpoint(tmp_path / "ck.bin")
        s.run(5)
        after = s.fields()
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel) as s:
        s.restore(tmp_path / "ck.bin")
        assert all(np.array_equal(_bits(s.field(k)), _bits(v)) for k, v in want.items())
        s.run(5)
        assert all(np.array_equal(_bits(s.field(k)), _bits(v)) for k, v in after.items())
    if kernel == fg.KERNEL_TWO_PASS:
        return  # no batch form
    b = fg.Batch(0, kernel)
    sid = b.add(p, codes, specs, steps + 5, scheme=fg.SCHEME_CORRECTED)
    b.run(steps + 5)
    got = b.fields(sid)
    name = "ey"
    b.done(b.read_async(sid, name, pinned.view(codes.shape)), wait=True)
    assert np.array_equal(_bits(pinned.view(codes.shape)), _bits(got[name]))
    b.done(b.read_async(sid, name, pinned.view((1, ny, nx)), z0=nz // 2, nplanes=1), wait=True)
    assert np.array_equal(_bits(pinned.view((1, ny, nx))[0]), _bits(got[name][nz // 2]))
    b.close()
    assert all(np.array_equal(_bits(got[k]), _bits(v)) for k, v in after.items())


def test_read_longer_than_the_staging_area(cuda):
    # 5.2 M cells: two pieces of 4 M floats, the border inside a row
    dims = (217, 155, 155)
    codes, specs, _, sources, consts, jz = random_case(8, 8, 8, seed=1, ncls=2, nsrc=1)
    codes = np.zeros(dims[::-1], np.uint8)
    p = Params(make_params(dims, consts, [(100, 70, 70)], jz))
    pinned = fg.PinnedBuffer(codes.size)
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED) as s:
        s.run(90)
        a = s.field("ez")
        b = s.field("ez", out=pinned.view(codes.shape))
        assert np.any(a[:40]) and np.any(a[-40:])
        assert np.array_equal(_bits(a), _bits(b))


@pytest.mark.parametrize("dims", [(3, 5, 4), (4, 3, 5), (16, 9, 7), (17, 9, 6), (33, 10, 5), (64, 21, 19), (257, 67, 41)])
def test_reads_land_on_any_alignment_and_nowhere_else(cuda, dims):
    """Page-locked destinations at every offset from a 16-byte boundary (the
    kernel writes 16 bytes at a time, its first and last group partly) and off
    a float's own alignment, dense and padded rows: the values are those of a
    pageable read, and the elements around the volume are not touched."""
    torch, (nx, ny, nz) = cuda, dims
    codes, specs, _, sources, consts, jz = random_case(*dims, seed=7, ncls=3, nsrc=2)
    p = Params(make_params(dims, consts, sources, jz))
    n, guard = nx * ny * nz, 8
    raw = torch.zeros(4 * (n + 2 * guard) + 16, dtype=torch.uint8, pin_memory=True).numpy()
    with fg.Solver(p, codes, specs, scheme=fg.SCHEME_CORRECTED) as s:
        s.run(8)
        want = s.field("ez")
        assert np.count_nonzero(want)
        for skew in (0, 4, 8, 12, 2):  # bytes
            raw[:] = 0xA5
            lo = 4 * guard + skew
            out = raw[lo:lo + 4 * n].view(np.float32).reshape(codes.shape)
            s.field("ez", out=out)
            assert out.tobytes() == want.tobytes(), skew
            assert np.all(raw[:lo] == 0xA5) and np.all(raw[lo + 4 * n:] == 0xA5), skew
