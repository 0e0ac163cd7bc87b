"""Timed cases of the framework: what a user has it do, through its public
entry points.

A case is a plain dict.  ``entry`` names the way in:

  solver     one resident solve (Solver): run some steps, read E to the host
  monitored  the same with probes and a running DFT installed, read at the end
  solve      a whole solve: create, run, read, close (a new geometry per call)
  native     Plan + fdtd_step (or fdtd_step_h / fdtd_step_de) on the caller's
             own device buffers
  compat     the five reference kernels' launchers on the caller's buffers
  batch      many uneven solves advanced together (Batch), fields read through
             page-locked memory

``form`` is the stored state: d (every field), two_pass, compact, compact16.
Grids hold nested Debye ellipsoids in vacuum with a z dipole outside them and
Mur faces; the corrected scheme at 0.99 of the Courant limit, except through
the compat launchers, which have the reference's scheme only.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

import fdtd_gb300 as fg

FORMS = {"d": fg.KERNEL_SINGLE_PASS, "two_pass": fg.KERNEL_TWO_PASS, "compact": fg.KERNEL_COMPACT,
         "compact16": fg.KERNEL_COMPACT_R16}
# bytes a cell-update cannot do without: H, E and the Debye history read and
# written once, one class byte (history only on cells that have any: see work)
STATE_BYTES = {"d": (97, 0), "two_pass": (97, 0), "compact": (49, 24), "compact16": (49, 12.25)}
FLOPS = 60.0
TISSUE = 0.36      # share of the cells inside the outer ellipsoid, as in the benchmark's phantom
MOST = 512 * 512 * 400 * 60  # cell-updates of the largest listed case


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the plain 64^3 sphere-sized problem: launches and latency, state inside L2
        dict(name="solver_64_d", entry="solver", form="d", nx=64, ny=64, nz=64, steps=200),
        # the benchmark's voxel phantom, every field kept
        dict(name="phantom_512_d", entry="solver", form="d", nx=512, ny=512, nz=400, steps=60),
        # the same in the reduced-storage form
        dict(name="phantom_512_r16", entry="solver", form="compact16", nx=512, ny=512, nz=400, steps=60),
        # a head-sized voxel model: none of its sizes a multiple of anything
        dict(name="head_odd_d", entry="solver", form="d", nx=217, ny=253, nz=181, steps=60),
        dict(name="head_odd_compact", entry="solver", form="compact", nx=301, ny=245, nz=187, steps=60),
        # a dosimetry run: probe series, running DFT, peak SAR
        dict(name="monitored_compact", entry="monitored", form="compact", nx=224, ny=208, nz=176, steps=120),
        # one request of a stream of geometries, start to end
        dict(name="solve_r16", entry="solve", form="compact16", nx=150, ny=134, nz=170, steps=300),
        # the reference program with its kernels swapped for the launchers: one step
        dict(name="compat_256", entry="compat", form="d", nx=256, ny=256, nz=200, steps=1),
        dict(name="compat_small", entry="compat", form="d", nx=61, ny=52, nz=47, steps=1),
        # a caller that owns its device memory: fused steps on dense odd rows
        dict(name="native_odd", entry="native", form="d", nx=250, ny=239, nz=160, steps=4),
        # many small solves in one launch, every field kept
        dict(name="batch_small_d", entry="batch", form="d", lo=24, hi=128, solves=20, steps=48),
        # the batched workload's sizes in the reduced-storage form
        dict(name="batch_r16", entry="batch", form="compact16", lo=48, hi=256, solves=20, steps=48),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["solver", "solver", "solver", "monitored", "solve", "compat", "native", "batch"])
    if entry == "batch":
        lo = rng.randint(20, 64)
        hi = rng.randint(lo + 32, 256)
        case = dict(entry="batch", form=rng.choice(["d", "compact", "compact16"]), lo=lo, hi=hi,
                    solves=rng.randint(3, 20), steps=rng.choice([24, 48]))
        while case["solves"] > 3 and case["steps"] * sum(a * b * c for a, b, c in _batch_dims(case)) > MOST:
            case["solves"] -= 1
        return case
    while True:
        nx, ny, nz = (_log_uniform(rng, 24, m) for m in (512, 512, 400))
        if rng.random() < 0.4:
            nx = (nx + 15) // 16 * 16
        cells = nx * ny * nz
        if cells <= 512 * 512 * 400:
            break
    if entry == "compat":
        form, steps = "d", 1
    elif entry == "native":
        form, steps = rng.choice(["d", "d", "two_pass"]), 4
    else:
        form = rng.choice(["d", "compact", "compact16"] + (["two_pass"] if entry == "solver" else []))
        steps = max(30, min(240, MOST // cells // 4))
        steps = steps if entry == "solve" else steps // 2 * 2
    return dict(entry=entry, form=form, nx=nx, ny=ny, nz=nz, steps=steps)


# ----------------------------------------------------------------- inputs

class _Params:
    """An FdtdParams built in memory (its arrays are kept here)."""

    def __init__(self, dims, sources, jz):
        f32 = np.float32
        raw = fg.FdtdParams()
        raw.nx, raw.ny, raw.nz = dims
        raw.c = 299792458.0
        raw.pi = math.pi
        raw.waveFrequency = 1.0e9
        raw.pulseWidth, raw.pulseModulationFrequency, raw.elementsPerWave = 0.5, 0.9, 300
        raw.dx = raw.dy = raw.dz = 1.0e-3
        raw.dt = float(f32(0.99 * 1.0e-3 / (299792458.0 * math.sqrt(3.0))))
        raw.mu0 = 4e-7 * math.pi
        raw.eps0 = 8.8541878e-12
        raw.timeskip = 0.99
        raw.defaultSigma, raw.defaultEpsS, raw.defaultEpsI, raw.defaultTauD = 0.0, 1.0, 1.0, 0.0
        self._src = (C.c_int * (3 * len(sources)))(*[v for s in sources for v in s])
        self._jz = np.ascontiguousarray(jz, f32)
        raw.sourcesCount = len(sources)
        raw.sources = C.cast(self._src, C.POINTER(C.c_int))
        raw.jzCount = self._jz.size
        raw.jz = self._jz.ctypes.data_as(C.POINTER(C.c_float))
        self.raw = raw

    def __getattr__(self, name):
        return getattr(self.raw, name)

    @property
    def shape(self):
        return (self.raw.nz, self.raw.ny, self.raw.nx)


class _Problem:
    """Geometry, materials and source of one grid, from a seed alone.  The
    compat launchers' sources live in one block per device, so two problems
    that take turns there share them (fixed_source)."""

    def __init__(self, dims, seed, fixed_source=False):
        rng = random.Random(seed)
        self.dims = dims
        nx, ny, nz = dims
        shells = rng.randint(4, 8)
        self.specs = np.zeros((shells + 1, 4), np.float32)  # sigma, eps_s, eps_inf, tau; class 0 is vacuum
        self.specs[0] = (0.0, 1.0, 1.0, 0.0)
        for k in range(1, shells + 1):
            eps_i = rng.uniform(4, 40)
            self.specs[k] = (rng.uniform(0.05, 2.0), rng.uniform(max(eps_i, 10), 80), eps_i, rng.uniform(5e-12, 15e-12))
        outer = 2.0 * (TISSUE * 3.0 / (4.0 * math.pi)) ** (1.0 / 3.0)  # semi-axes over half the grid
        self.axes = [[n / 2 * outer * (1.0 - 0.8 * k / shells) * rng.uniform(0.95, 1.05) for n in dims]
                     for k in range(shells)]
        if fixed_source:
            rng = random.Random(1)
        # a three-cell z dipole near a low corner, where the ellipsoids do not reach
        at = [min(n - 3, max(2, int(n * rng.uniform(0.06, 0.16)))) for n in dims]
        self.sources = [(at[0], at[1], at[2] + d) for d in (-1, 0, 1)]
        f = rng.uniform(0.3e9, 3e9)
        n = np.arange(fg.JZ_LEN)
        dt = 0.99 * 1.0e-3 / (299792458.0 * math.sqrt(3.0))
        self.jz = (1e-3 * np.sin(2 * math.pi * f * n * dt) * (1 - np.exp(-n / 20.0))).astype(np.float32)
        self.probes = [(rng.randrange(nx), rng.randrange(ny), rng.randrange(nz)) for _ in range(12)] + \
                      [self.sources[0]]
        self.params = _Params(dims, self.sources, self.jz)
        self._classes()

    def _classes(self):
        dev = "cuda"
        nx, ny, nz = self.dims
        ax = [(torch.arange(n, device=dev, dtype=torch.float32) - (n - 1) / 2) for n in self.dims]
        codes = torch.zeros((nz, ny, nx), dtype=torch.uint8, device=dev)
        for k, (a, b, c) in enumerate(self.axes):
            yz = (ax[2] / c).square()[:, None] + (ax[1] / b).square()[None, :]
            codes[yz[:, :, None] + (ax[0] / a).square() <= 1.0] = k + 1
        self.codes_dev = codes
        self.codes = codes.cpu().numpy()


def _randoms(shape, seed, count, scale):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [torch.randn(shape, device="cuda", generator=g) * s for s in scale for _ in range(count)]


def _pinned(shape):
    """Three page-locked field volumes to read into."""
    return [torch.zeros(shape, dtype=torch.float32, pin_memory=True).numpy() for _ in range(3)]


def _batch_dims(case):
    # the sizes belong to the case, the geometry to the seed
    rng = random.Random(case["lo"] * 1000003 + case["hi"])
    return [tuple(_log_uniform(rng, case["lo"], case["hi"]) for _ in range(3)) for _ in range(case["solves"])]


E_SCALE, H_SCALE, D_SCALE = 1.0, 1.0 / 377.0, 8.85e-12


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    entry, kernel = case["entry"], FORMS[case["form"]]
    if entry == "batch":
        s.batch = fg.Batch(0, kernel)
        s.ids, s.out = [], []
        for k, dims in enumerate(_batch_dims(case)):
            q = _Problem(dims, seed * 131 + k)
            s.ids.append(s.batch.add(q.params, q.codes, q.specs, 1 << 30, scheme=fg.SCHEME_CORRECTED))
            s.out.append(_pinned(q.params.shape))
        return s
    s.problem = q = _Problem((case["nx"], case["ny"], case["nz"]), seed, fixed_source=entry == "compat")
    shape = q.params.shape
    if entry in ("solver", "monitored"):
        s.solver = fg.Solver(q.params, q.codes, q.specs, scheme=fg.SCHEME_CORRECTED, kernel=kernel)
        if entry == "monitored":
            s.solver.set_probes(q.probes, capacity=case["steps"])
            s.solver.set_dft(0.9e9, stride=5, z0=shape[0] // 4, nplanes=max(1, shape[0] // 8))
    if entry in ("solver", "monitored", "solve"):
        s.out = _pinned(shape)
        return s
    # the caller's own device buffers
    s.lib = fg.lib()
    s.stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if entry == "native":
        s.plan = fg.Plan(q.params, q.specs, scheme=fg.SCHEME_CORRECTED)
        t = _randoms(shape, seed, 3, (H_SCALE, H_SCALE, E_SCALE, E_SCALE, D_SCALE, D_SCALE))
        two = case["form"] == "two_pass"
        if not two:
            t[3:6] = [v.clone() for v in t[0:3]]  # both H buffers hold the same untouched cells
        s.h, s.e, s.d = [t[0:3], t[0:3] if two else t[3:6]], [t[6:9], t[9:12]], [t[12:15], t[15:18]]
        s.n = 0
        s.fields = []
        for n in range(2):
            f = fg.NativeFields()
            cur, prv = (n + 1) % 2, n % 2
            for k, c in enumerate("xyz"):
                setattr(f, "h" + c, s.h[n][k].data_ptr())
                setattr(f, "h" + c + "_out", s.h[(n + 1) % 2][k].data_ptr())
                setattr(f, "e" + c, s.e[cur][k].data_ptr())
                setattr(f, "e" + c + "_prev", s.e[prv][k].data_ptr())
                setattr(f, "d" + c, s.d[cur][k].data_ptr())
                setattr(f, "d" + c + "_prev", s.d[prv][k].data_ptr())
            f.material = q.codes_dev.data_ptr()
            s.fields.append(f)
        return s
    # compat: three E and three D slots, per-cell material arrays, Mur slabs
    fg.check(s.lib.fdtd_copy_symbols(C.byref(q.params.raw)), "fdtd_copy_symbols")
    t = _randoms(shape, seed, 3, (H_SCALE, E_SCALE, E_SCALE, D_SCALE, D_SCALE))
    s.h, s.e1, s.e2, s.d1, s.d2 = (t[3 * k:3 * k + 3] for k in range(5))
    s.e0 = [torch.zeros_like(v) for v in s.h]
    s.d0 = [torch.zeros_like(v) for v in s.h]
    table = torch.from_numpy(q.specs).cuda()
    idx = q.codes_dev.long()
    s.media = [table[:, k][idx].contiguous() for k in (0, 2, 1, 3)]  # sigma, eps_inf, eps_s, tau
    del idx
    s.rp = [torch.ones(v, device="cuda") for v in fg.rp_shapes(case["nx"], case["ny"], case["nz"])]
    return s


def _ptrs(tensors):
    return [C.c_void_p(t.data_ptr()) for t in tensors]


def run(s):
    case = s.case
    entry, steps = case["entry"], case["steps"]
    if entry == "batch":
        s.batch.run(steps)
        tickets = [s.batch.read_async(i, "e" + c, out[k]) for i, out in zip(s.ids, s.out) for k, c in enumerate("xyz")]
        for t in tickets:
            s.batch.done(t, wait=True)
        return s.out
    if entry == "solver":
        s.solver.run(steps)
        return [s.solver.field("e" + c, out=s.out[k]) for k, c in enumerate("xyz")]
    if entry == "monitored":
        s.solver.run(steps)
        peak, _ = s.solver.peak_sar()
        return {"probes": s.solver.probes(), "peak_sar": peak, "dft_z": s.solver.dft(2),
                "ez": s.solver.field("ez", out=s.out[2])}
    if entry == "solve":
        q = s.problem
        with fg.Solver(q.params, q.codes, q.specs, scheme=fg.SCHEME_CORRECTED, kernel=FORMS[case["form"]]) as solver:
            solver.run(steps)
            return [solver.field("e" + c, out=s.out[k]) for k, c in enumerate("xyz")]
    L = s.lib
    if entry == "native":
        for _ in range(steps):
            f = C.byref(s.fields[s.n & 1])
            if case["form"] == "two_pass":
                fg.check(L.fdtd_step_h(s.plan.handle, f, s.stream), "fdtd_step_h")
                fg.check(L.fdtd_step_de(s.plan.handle, f, s.n, s.stream), "fdtd_step_de")
            else:
                fg.check(L.fdtd_step(s.plan.handle, f, s.n, s.stream), "fdtd_step")
            s.n += 1
        k = (s.n - 1) & 1
        return {"h": s.h[s.n & 1], "e": s.e[k], "d": s.d[k]}
    # the reference's loop body (its argument order), step index 3
    h, e0, e1, e2 = _ptrs(s.h), _ptrs(s.e0), _ptrs(s.e1), _ptrs(s.e2)
    d0, d1, d2 = _ptrs(s.d0), _ptrs(s.d1), _ptrs(s.d2)
    st = s.stream
    fg.check(L.fdtd_update_h(*h, *e2, st), "fdtd_update_h")
    fg.check(L.fdtd_update_d(*d0, *d2, *h, st), "fdtd_update_d")
    fg.check(L.fdtd_update_sources(d0[2], d2[2], h[0], h[1], 3, st), "fdtd_update_sources")
    fg.check(L.fdtd_update_e(*e0, *e2, *e1, *d0, *d2, *d1, *_ptrs(s.media), st), "fdtd_update_e")
    fg.check(L.fdtd_update_mur(*e0, *e2, *_ptrs(s.rp), st), "fdtd_update_mur")
    return {"h": s.h, "d": s.d0, "e": s.e0}


# ------------------------------------------------------------------- work

def work(case):
    if case["entry"] == "batch":
        cells = sum(a * b * c for a, b, c in _batch_dims(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    dense, history = STATE_BYTES[case["form"]]
    updates = cells * case["steps"]
    per = dense + history * TISSUE
    if case["entry"] == "compat":  # H, D and E each read and written by their own kernel, four float materials
        per = 4.0 * (3 + 3 + 3 + 3 + 3 + 3 + 3 + 12 + 4 + 3)
    if case["form"] == "two_pass":
        per = 121.0
    total = per * updates
    if case["entry"] in ("solver", "solve", "batch"):
        total += 12.0 * cells  # E read out
    if case["entry"] == "monitored":
        total += 4.0 * cells + (case["steps"] // 5) * 108.0 * cells / 8
    return {"bytes": float(total), "flops": FLOPS * updates}


# ------------------------------------------------------- the 64-bit answer

def _mur(t, s, consts):
    """First-order Mur on the faces, vacuum slabs; the corrected scheme's far
    ey face unless consts says otherwise."""
    dt, q = consts["dt"], consts["dx"] * math.sqrt(consts["mu0"] * consts["eps0"])

    def value(tn, sn, sf):
        return ((dt - q) * tn + (dt + q) * sn - (dt - q) * sf) / (dt + q)

    def face(k, axis, lo, ranges, old=False):
        at, nb = (0, 1) if lo else (-1, -2)
        i = [slice(None)] * 3
        for a, r in ranges.items():
            i[a] = r
        f, g = list(i), list(i)
        f[axis], g[axis] = at, nb
        f, g = tuple(f), tuple(g)
        t[k][f] = value((s if old else t)[k][g], s[k][g], s[k][f])

    mid, head, inner = slice(1, -1), slice(0, -1), slice(1, -1)
    for lo in (True, False):
        face(0, 1, lo, {0: mid, 2: head})
        face(0, 0, lo, {1: mid, 2: head})
        face(1, 2, lo, {0: mid, 1: head}, old=not lo and not consts["corrected"])
        face(1, 0, lo, {1: head, 2: inner})
        face(2, 2, lo, {0: head, 1: mid})
        face(2, 1, lo, {0: head, 2: inner})


def _update_h(h, e, k):
    (hx, hy, hz), (ex, ey, ez) = h, e
    hx[:-1, :-1, 1:-1] += k * ((ey[1:, :-1, 1:-1] - ey[:-1, :-1, 1:-1]) - (ez[:-1, 1:, 1:-1] - ez[:-1, :-1, 1:-1]))
    hy[:-1, 1:-1, :-1] += k * ((ez[:-1, 1:-1, 1:] - ez[:-1, 1:-1, :-1]) - (ex[1:, 1:-1, :-1] - ex[:-1, 1:-1, :-1]))
    hz[1:-1, :-1, :-1] += k * ((ex[1:-1, 1:, :-1] - ex[1:-1, :-1, :-1]) - (ey[1:-1, :-1, 1:] - ey[1:-1, :-1, :-1]))


def _update_d(t, s, h, k, sources, jz):
    hx, hy, hz = h
    t[0][1:-1, 1:-1, :-1] = s[0][1:-1, 1:-1, :-1] + k * (
        (hz[1:-1, 1:-1, :-1] - hz[1:-1, :-2, :-1]) - (hy[1:-1, 1:-1, :-1] - hy[:-2, 1:-1, :-1]))
    t[1][1:-1, :-1, 1:-1] = s[1][1:-1, :-1, 1:-1] + k * (
        (hx[1:-1, :-1, 1:-1] - hx[:-2, :-1, 1:-1]) - (hz[1:-1, :-1, 1:-1] - hz[1:-1, :-1, :-2]))
    t[2][:-1, 1:-1, 1:-1] = s[2][:-1, 1:-1, 1:-1] + k * (
        (hy[:-1, 1:-1, 1:-1] - hy[:-1, 1:-1, :-2]) - (hx[:-1, 1:-1, 1:-1] - hx[:-1, :-2, 1:-1]))
    for x, y, z in sources:
        t[2][z, y, x] = s[2][z, y, x] + k * ((hy[z, y, x] - hy[z, y, x - 1]) - (hx[z, y, x] - hx[z, y - 1, x])) - jz


def _update_e(t, e0, e1, d0, d1, d2, coef, consts):
    a, c, d, tau = coef
    dt = consts["dt"]
    for k in range(3):
        i = (slice(1, -1), slice(1, -1), slice(0, -1)) if k == 0 else (slice(1, None), slice(None), slice(1, None))
        g1, g2 = d0[k][i] - d1[k][i], d1[k][i] - d2[k][i]
        t[k][i] = c[i] * (d[i] * e0[k][i] - a[i] * e1[k][i] + 2 * dt * g1 + 2 * tau[i] * (g1 - g2))


def _coefs(q, consts):
    sig, es, ei, tau = (torch.from_numpy(q.specs[:, k].astype(np.float64)).cuda() for k in range(4))
    dt, eps0 = consts["dt"], consts["eps0"]
    a = 2 * eps0 * ei * tau
    b = a + 2 * dt * (eps0 * es + sig * tau)
    c = 1 / (b + sig * dt * dt)
    d = (a + b if consts["corrected"] else 2 * b) - sig * dt * dt
    idx = q.codes_dev.long()
    return [v[idx] for v in (a, c, d, tau)]


def _consts(q, corrected):
    r = q.params.raw
    return {"dt": r.dt, "dx": r.dx, "mu0": r.mu0, "eps0": r.eps0, "corrected": corrected}


def _simulate(q, steps, h, e, d, each=None):
    """`steps` steps from h, e = [slot][component], d likewise (float64, as the
    native path's slots: step n writes slot n % 2)."""
    k = _consts(q, True)
    kh, kd = k["dt"] / (k["mu0"] * k["dx"]), k["dt"] / k["dx"]
    coef = _coefs(q, k)
    for n in range(steps):
        cur, prv = (n + 1) % 2, n % 2
        _update_h(h, e[cur], kh)
        dn = [v.clone() for v in d[prv]]
        _update_d(dn, d[cur], h, kd, q.sources, float(q.jz[n]))
        en = [v.clone() for v in e[prv]]
        _update_e(en, e[cur], e[prv], dn, d[cur], d[prv], coef, k)
        _mur(en, e[cur], k)
        e[prv], d[prv] = en, dn
        if each is not None:
            each(n, en)
    return h, e[(steps - 1) % 2], d[(steps - 1) % 2]


def _from_rest(q, steps, each=None):
    def zeros():
        return [torch.zeros(q.params.shape, dtype=torch.float64, device="cuda") for _ in range(3)]

    return _simulate(q, steps, zeros(), [zeros(), zeros()], [zeros(), zeros()], each)


def exact(case, seed):
    entry, steps = case["entry"], case["steps"]
    if entry == "batch":
        out = []
        for k, dims in enumerate(_batch_dims(case)):
            e = _from_rest(_Problem(dims, seed * 131 + k), steps)[1]
            out.append([v.cpu().numpy() for v in e])
        return out
    q = _Problem((case["nx"], case["ny"], case["nz"]), seed, fixed_source=entry == "compat")
    shape = q.params.shape
    if entry in ("solver", "solve"):
        return _from_rest(q, steps)[1]
    if entry == "monitored":
        dt, w = q.params.raw.dt, 2 * math.pi * 0.9e9
        z0, planes = shape[0] // 4, max(1, shape[0] // 8)
        acc = [torch.zeros((planes,) + shape[1:], dtype=torch.complex128, device="cuda") for _ in range(3)]
        series = torch.zeros((steps, len(q.probes), 3), dtype=torch.float64, device="cuda")
        px, py, pz = (torch.tensor([p[k] for p in q.probes], device="cuda") for k in range(3))

        def each(n, e):
            for c in range(3):
                series[n, :, c] = e[c][pz, py, px]
                if (n + 1) % 5 == 0:
                    t = (n + 1) * dt
                    acc[c] += e[c][z0:z0 + planes] * (complex(math.cos(w * t), -math.sin(w * t)) * 5 * dt)

        e = _from_rest(q, steps, each)[1]
        sigma = torch.from_numpy(q.specs[:, 0].astype(np.float64)).cuda()[q.codes_dev[z0:z0 + planes].long()]
        sar = sigma * sum(v.abs().square() for v in acc) / 2000.0
        return {"probes": series, "peak_sar": float(sar.max()), "dft_z": acc[2].cpu().numpy(), "ez": e[2]}
    if entry == "native":
        t = [v.double() for v in _randoms(shape, seed, 3, (H_SCALE, H_SCALE, E_SCALE, E_SCALE, D_SCALE, D_SCALE))]
        h, e, d = _simulate(q, steps, t[0:3], [t[6:9], t[9:12]], [t[12:15], t[15:18]])
        return {"h": h, "e": e, "d": d}
    k = _consts(q, False)
    t = [v.double() for v in _randoms(shape, seed, 3, (H_SCALE, E_SCALE, E_SCALE, D_SCALE, D_SCALE))]
    h, e1, e2, d1, d2 = (t[3 * j:3 * j + 3] for j in range(5))
    e0 = [torch.zeros_like(v) for v in h]
    d0 = [torch.zeros_like(v) for v in h]
    _update_h(h, e2, k["dt"] / (k["mu0"] * k["dx"]))
    _update_d(d0, d2, h, k["dt"] / k["dx"], q.sources, float(q.jz[3]))
    _update_e(e0, e2, e1, d0, d2, d1, _coefs(q, k), k)
    _mur(e0, e2, k)
    return {"h": h, "d": d0, "e": e0}
