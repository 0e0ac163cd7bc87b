// device_common.cuh -- device helpers shared by the compat and native kernels.
#pragma once

#include <cuda_runtime.h>

#include "fdtd_internal.h"

namespace fdtd {

__host__ __device__ inline size_t cell_index(int x, int y, int z, int nx, int ny)
{
    return ((size_t)z * (size_t)ny + (size_t)y) * (size_t)nx + (size_t)x;
}

// Tile of a block in a grid of (tiles in x * tiles in y, z) blocks, x fastest:
// flat, as gridDim.y's limit of 65535 is too low for tiles of a few rows.
struct TileXY {
    int x0, y0;
    __device__ __forceinline__ TileXY(int nx, int tx, int ty)
    {
        const unsigned tiles = (unsigned)(nx + tx - 1) / tx, by = blockIdx.x / tiles;
        x0 = (int)(blockIdx.x - by * tiles) * tx;
        y0 = (int)by * ty;
    }
};

inline dim3 tile_grid(int nx, int ny, int nz, int tx, int ty, int tz)
{
    return dim3((unsigned)((nx + tx - 1) / tx) * (unsigned)((ny + ty - 1) / ty), (unsigned)((nz + tz - 1) / tz));
}

// Programmatic dependent launch: lets the next launch's blocks be placed while
// this grid finishes, and (before any access to memory) waits for the previous
// grid to complete.  A stream's order is kept: every kernel launched this way
// waits before it reads or writes.  Such a kernel's lifetime begins before the
// previous grid has ended, so none of its parameters is a const __restrict__
// pointer: loads of data said to be constant for the kernel's lifetime may take
// the read-only path, or move ahead of the wait.
__device__ __forceinline__ void pdl_begin()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Whether stream is being captured (an error is left to the launch to report).
inline bool capturing(cudaStream_t stream)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return status != cudaStreamCaptureStatusNone;
}

// Launches kernel so that its blocks may be placed before the stream's
// previous grid completes; the kernel must call pdl_begin() first.  In a
// caller's capture the launch is a plain one, unless own_graph says that the
// graph is this library's: a graph with programmatic edges cannot be read by
// code that knows plain ones (cudaGraphGetEdges without edge data fails).
template <class... P, class... A>
int launch_pdl(bool own_graph, void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t stream, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = own_graph || !capturing(stream) ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e != cudaSuccess)
        cudaGetLastError();  // reported here, not by a later call too
    return e == cudaSuccess ? FDTD_OK : (int)e;
}

// updateHField (fdtd_calculations.cu:32-77) for the cells (x, y, z0 .. z0+K-1),
// x < nx-1, y < ny-1: every load before the first store, and E^n x, y of a
// plane read once for the cells below and above it.  out may be in.
template <int K>
__device__ __forceinline__ void h_column(int x, int y, int z0, int nx, int ny, int nz, int pitch, float kx, float ky,
                                         float kz, const float *ex, const float *ey, const float *ez,
                                         const float *const in[3], float *const out[3])
{
    const int n = min(K, nz - 1 - z0);  // no component is updated at z = nz-1
    const size_t i = cell_index(x, y, z0, pitch, ny), sy = pitch, sz = (size_t)pitch * ny;
    const bool xi = x >= 1, yi = y >= 1;
    float a[K + 1], b[K + 1], c[K], ay[K], bx[K], cx[K], cy[K], h[3][K];
#pragma unroll
    for (int k = 0; k <= K; k++)
        if (k <= n) {
            a[k] = ex[i + k * sz];
            b[k] = ey[i + k * sz];
        }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (k < n) {
            const size_t j = i + k * sz;
            c[k] = ez[j];
            cy[k] = ez[j + sy];
            cx[k] = ez[j + 1];
            ay[k] = ex[j + sy];
            bx[k] = ey[j + 1];
            h[0][k] = in[0][j];
            h[1][k] = in[1][j];
            h[2][k] = in[2][j];
        }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (k < n) {
            const size_t j = i + k * sz;
            // hx: both terms scaled by dy (fdtd_calculations.cu:48-52)
            if (xi)
                out[0][j] = h[0][k] - ky * (cy[k] - c[k]) + ky * (b[k + 1] - b[k]);
            if (yi)
                out[1][j] = h[1][k] - kz * (a[k + 1] - a[k]) + kx * (cx[k] - c[k]);
            if (z0 + k >= 1)
                out[2][j] = h[2][k] - kx * (bx[k] - b[k]) + ky * (ay[k] - a[k]);
        }
}

// Debye E update of one component (fdtd_calculations.cu:150-156): E^{n+1} =
// c (d E^n - a E^{n-1} + k1 D^{n+1} - k2 D^n + k3 D^{n-1}), the D terms in
// the difference form of DebyeCoef.
__device__ __forceinline__ float debye_update(const DebyeCoef &k, float e0, float e1, float d0, float d1, float d2)
{
    const float p = k.d * e0 - k.a * e1;
    const float g1 = d0 - d1;
    const float g2 = d1 - d2;
    const float q = k.two_dt * g1 + k.two_tau * (g1 - g2) + k.delta * d0;
    return k.c * (p + q);
}

// The reference's per-cell coefficients (fdtd_calculations.cu:141-144) in
// single precision.  The reference evaluates a, b, c, d with double literals;
// here c is the correctly rounded reciprocal of the same float sum, d is the
// same single rounding, a and b may differ from it by one unit in the last
// place.  delta comes from an exact two-sum of dt + tau.  Where the products
// of b fuse is written out: left to the compiler it changed with the order of
// the kernel's loads, and with it the last bit for one material in three (the
// other order of fusing was up to 3 % further from 64 bits).
__device__ __forceinline__ DebyeCoef cell_coef(float dt, float eps0, float sigma, float eps_s, float eps_i, float tau,
                                               int scheme)
{
    DebyeCoef k;
    const float a = 2.0f * eps0 * eps_i * tau;
    const float x = __fmaf_rn(eps0, eps_s, __fmul_rn(sigma, tau));
    const float b = __fmaf_rn(__fmul_rn(2.0f, dt), x, a);
    const float s = __fmul_rn(__fmul_rn(sigma, dt), dt);
    k.a = a;
    k.c = __frcp_rn(__fadd_rn(b, s));
    k.d = scheme == FDTD_SCHEME_CORRECTED ? __fsub_rn(__fadd_rn(a, b), s) : __fsub_rn(2.0f * b, s);
    k.two_dt = 2.0f * dt;
    k.two_tau = 2.0f * tau;
    const float sum = __fadd_rn(dt, tau);
    const float bb = __fsub_rn(sum, dt);
    const float err = __fadd_rn(__fsub_rn(dt, __fsub_rn(sum, bb)), __fsub_rn(tau, bb));
    k.delta = -2.0f * err;
    k.pad0 = k.pad1 = 0.0f;
    return k;
}

// First-order Mur value of one face cell (fdtd_calculations.cu:240-248 and
// mirrors).  rp_self is the slab layer on the face, rp_nbr one cell inwards;
// t_nbr is E^{n+1} at the inner neighbour, s_nbr and s_self are E^n.
__device__ __forceinline__ float mur_value(float dt, float h, float me, float rp_self, float rp_nbr, float t_nbr,
                                           float s_nbr, float s_self)
{
    // every operation rounded on its own, in the reference's order
    // (fdtd_calculations.cu:240-247): no contraction into fused multiply-adds,
    // so each kernel that applies a Mur face gets the same bits
    const float q_self = __fmul_rn(h, sqrtf(__fmul_rn(me, rp_self)));
    const float q_nbr = __fmul_rn(h, sqrtf(__fmul_rn(me, rp_nbr)));
    const float num = __fsub_rn(__fadd_rn(__fmul_rn(__fsub_rn(dt, q_nbr), t_nbr), __fmul_rn(__fadd_rn(dt, q_nbr), s_nbr)),
                                __fmul_rn(__fsub_rn(dt, q_self), s_self));
    return __fmul_rn(__fdiv_rn(1.0f, __fadd_rn(dt, q_self)), num);
}

// mur_value of a face cell whose slab layers hold one value, from that
// value's factors k = (1/(dt+q), dt-q, dt+q, dt-q): the same operations on
// the same operands, so the same bits.
__device__ __forceinline__ float mur_value_k(float4 k, float t_nbr, float s_nbr, float s_self)
{
    return __fmul_rn(k.x, __fsub_rn(__fadd_rn(__fmul_rn(k.y, t_nbr), __fmul_rn(k.z, s_nbr)), __fmul_rn(k.w, s_self)));
}

// The twelve (component, face) sets that updateMurBoundary writes.  For face
// set f, (len_u, len_v) is the extent and (u0, v0) the first coordinate of
// its two in-face axes; `axis` is the face normal (0 x, 1 y, 2 z) and `far`
// selects the face at n-1.
struct MurFace {
    int comp, axis, far;
    int u0, len_u, v0, len_v;  // u is the faster in-face axis (x, else y)
};

__host__ __device__ inline MurFace mur_face(int f, int nx, int ny, int nz)
{
    MurFace m;
    m.comp = f / 4;
    m.far = f & 1;
    const int pair = (f >> 1) & 1;
    if (m.comp == 0) {          // ex: y faces (x 0..nx-2, z 1..nz-2), z faces (x 0..nx-2, y 1..ny-2)
        m.axis = pair ? 2 : 1;
        m.u0 = 0; m.len_u = nx - 1;
        if (m.axis == 1) { m.v0 = 1; m.len_v = nz - 2; }
        else { m.v0 = 1; m.len_v = ny - 2; }
    } else if (m.comp == 1) {   // ey: x faces (y 0..ny-2, z 1..nz-2), z faces (x 1..nx-2, y 0..ny-2)
        m.axis = pair ? 2 : 0;
        if (m.axis == 0) { m.u0 = 0; m.len_u = ny - 1; m.v0 = 1; m.len_v = nz - 2; }
        else { m.u0 = 1; m.len_u = nx - 2; m.v0 = 0; m.len_v = ny - 1; }
    } else {                    // ez: x faces (y 1..ny-2, z 0..nz-2), y faces (x 1..nx-2, z 0..nz-2)
        m.axis = pair ? 1 : 0;
        if (m.axis == 0) { m.u0 = 1; m.len_u = ny - 2; m.v0 = 0; m.len_v = nz - 1; }
        else { m.u0 = 1; m.len_u = nx - 2; m.v0 = 0; m.len_v = nz - 1; }
    }
    return m;
}

struct MurSlabs {
    const float *rpx0, *rpy0, *rpz0, *rpx_end, *rpy_end, *rpz_end;
};

// Applies updateMurBoundary to face set f, in-face position (iu, iv); pitch
// is the row stride of the E arrays (nx when dense).
// eT: E^{n+1} (written), eS: E^n.  fix_ey selects the corrected scheme's
// E^{n+1} term on the ey x = nx-1 face (the reference reads E^n there, :323).
__device__ __forceinline__ void mur_apply(int f, int iu, int iv, int nx, int ny, int nz, int pitch, float dt, float hx,
                                          float hy,
                                          float hz, float me, const MurSlabs &rp, float *t0, float *t1, float *t2,
                                          const float *s0, const float *s1, const float *s2, bool fix_ey)
{
    const MurFace m = mur_face(f, nx, ny, nz);
    if (iu >= m.len_u || iv >= m.len_v)
        return;
    const int u = m.u0 + iu, v = m.v0 + iv;
    int x, y, z, dxn = 0, dyn = 0, dzn = 0;
    float h, rs, rn;
    if (m.axis == 0) {
        x = m.far ? nx - 1 : 0; y = u; z = v; dxn = m.far ? -1 : 1; h = hx;
        const float *slab = m.far ? rp.rpx_end : rp.rpx0;
        const size_t base = ((size_t)z * ny + y) * 2;
        rs = slab[base + (m.far ? 1 : 0)];
        rn = slab[base + (m.far ? 0 : 1)];
    } else if (m.axis == 1) {
        x = u; y = m.far ? ny - 1 : 0; z = v; dyn = m.far ? -1 : 1; h = hy;
        const float *slab = m.far ? rp.rpy_end : rp.rpy0;
        rs = slab[((size_t)z * 2 + (m.far ? 1 : 0)) * nx + x];
        rn = slab[((size_t)z * 2 + (m.far ? 0 : 1)) * nx + x];
    } else {
        x = u; y = v; z = m.far ? nz - 1 : 0; dzn = m.far ? -1 : 1; h = hz;
        const float *slab = m.far ? rp.rpz_end : rp.rpz0;
        rs = slab[((size_t)(m.far ? 1 : 0) * ny + y) * nx + x];
        rn = slab[((size_t)(m.far ? 0 : 1) * ny + y) * nx + x];
    }
    const size_t i = cell_index(x, y, z, pitch, ny);
    const size_t j = cell_index(x + dxn, y + dyn, z + dzn, pitch, ny);
    // component pointers picked with selects (an indexed array would live in local memory)
    const float *S = m.comp == 0 ? s0 : (m.comp == 1 ? s1 : s2);
    float *T = m.comp == 0 ? t0 : (m.comp == 1 ? t1 : t2);
    // fdtd_calculations.cu:323: the ey face at x = nx-1 reads E^n at x-1 in
    // its first term as well.
    const bool quirk = m.comp == 1 && m.axis == 0 && m.far && !fix_ey;
    const float t_nbr = quirk ? S[j] : T[j];
    T[i] = mur_value(dt, h, me, rs, rn, t_nbr, S[j], S[i]);
}

// Indices of one face cell at face coordinates (u, v): the cell, its inward
// neighbour and its two Mur slab entries (self, neighbour).
struct MurCellIdx {
    size_t face, nbr, rs, rn;
};

__device__ __forceinline__ MurCellIdx mur_cell_idx(const MurFace &m, int u, int v, int nx, int ny, int nz, int pitch)
{
    const int ks = m.far ? 1 : 0, kn = m.far ? 0 : 1;
    int x, y, z, dxn = 0, dyn = 0, dzn = 0;
    MurCellIdx c;
    if (m.axis == 0) {
        x = m.far ? nx - 1 : 0; y = u; z = v; dxn = m.far ? -1 : 1;
        c.rs = ((size_t)z * ny + y) * 2 + ks;
        c.rn = ((size_t)z * ny + y) * 2 + kn;
    } else if (m.axis == 1) {
        x = u; y = m.far ? ny - 1 : 0; z = v; dyn = m.far ? -1 : 1;
        c.rs = ((size_t)z * 2 + ks) * nx + x;
        c.rn = ((size_t)z * 2 + kn) * nx + x;
    } else {
        x = u; y = v; z = m.far ? nz - 1 : 0; dzn = m.far ? -1 : 1;
        c.rs = ((size_t)ks * ny + y) * nx + x;
        c.rn = ((size_t)kn * ny + y) * nx + x;
    }
    c.face = cell_index(x, y, z, pitch, ny);
    c.nbr = cell_index(x + dxn, y + dyn, z + dzn, pitch, ny);
    return c;
}

// Operands of one face set: target / source arrays of its component, the
// array its neighbour term reads, its cell size and its slab.
struct MurSet {
    const MurFace m;
    float *T;
    const float *S, *TN, *slab;
    float h;
    __device__ __forceinline__ MurSet(int f, int nx, int ny, int nz, float hx, float hy, float hz, const MurSlabs &rp,
                                      float *t0, float *t1, float *t2, const float *s0, const float *s1,
                                      const float *s2, bool fix_ey)
        : m(mur_face(f, nx, ny, nz))
    {
        S = m.comp == 0 ? s0 : (m.comp == 1 ? s1 : s2);
        T = m.comp == 0 ? t0 : (m.comp == 1 ? t1 : t2);
        const bool quirk = m.comp == 1 && m.axis == 0 && m.far && !fix_ey;  // fdtd_calculations.cu:323
        TN = quirk ? S : T;
        h = m.axis == 0 ? hx : (m.axis == 1 ? hy : hz);
        slab = m.axis == 0 ? (m.far ? rp.rpx_end : rp.rpx0)
               : m.axis == 1 ? (m.far ? rp.rpy_end : rp.rpy0)
                             : (m.far ? rp.rpz_end : rp.rpz0);
    }
};

// mur_apply for K cells of one face set at in-face rows iv0, iv0 + vstride,
// ... below v_end: all loads are issued before any store, so K independent loads per
// array are in flight per thread (face cells are written, their neighbours
// and E^n are only read, so no cell is both).
// UNI: the set's slab holds one value whose factors are kf (no slab loads,
// no square roots or division).
template <int K, bool UNI = false>
__device__ __forceinline__ void mur_apply_k(int f, int iu, int iv0, int vstride, int v_end, int nx, int ny, int nz,
                                            int pitch,
                                            float dt, float hx, float hy, float hz, float me, const MurSlabs &rp,
                                            float *t0, float *t1, float *t2, const float *s0, const float *s1,
                                            const float *s2, bool fix_ey, float4 kf = float4{})
{
    const MurSet ms(f, nx, ny, nz, hx, hy, hz, rp, t0, t1, t2, s0, s1, s2, fix_ey);
    const MurFace &m = ms.m;
    if (iu >= m.len_u)
        return;
    const int u = m.u0 + iu;
    float rs[K], rn[K], tn[K], sn[K], sf[K];
    (void)rs;
    (void)rn;
    size_t face[K];
    bool on[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int iv = iv0 + k * vstride;
        on[k] = iv < m.len_v && iv < v_end;
        const MurCellIdx c = mur_cell_idx(m, u, m.v0 + (on[k] ? iv : 0), nx, ny, nz, pitch);
        face[k] = c.face;
        if (on[k]) {
            if constexpr (!UNI) {
                rs[k] = ms.slab[c.rs];
                rn[k] = ms.slab[c.rn];
            }
            tn[k] = ms.TN[c.nbr];
            sn[k] = ms.S[c.nbr];
            sf[k] = ms.S[c.face];
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (on[k]) {
            if constexpr (UNI)
                ms.T[face[k]] = mur_value_k(kf, tn[k], sn[k], sf[k]);
            else
                ms.T[face[k]] = mur_value(dt, ms.h, me, rs[k], rn[k], tn[k], sn[k], sf[k]);
        }
}

// mur_apply for K cells of one face set at flat in-face indices idx0,
// idx0 + stride, ... (row-major over (v, u), below len_u * len_v < 2^31);
// loads before stores as in mur_apply_k.
template <int K, bool UNI = false>
__device__ __forceinline__ void mur_apply_flat_k(int f, unsigned idx0, unsigned stride, int nx, int ny, int nz,
                                                 int pitch, float dt, float hx, float hy, float hz, float me,
                                                 const MurSlabs &rp, float *t0, float *t1, float *t2,
                                                 const float *s0, const float *s1, const float *s2, bool fix_ey,
                                                 unsigned limit = 0, float4 kf = float4{})
{
    const MurSet ms(f, nx, ny, nz, hx, hy, hz, rp, t0, t1, t2, s0, s1, s2, fix_ey);
    const MurFace &m = ms.m;
    if (m.len_u <= 0 || m.len_v <= 0)
        return;
    const unsigned lu = (unsigned)m.len_u;
    unsigned total = lu * (unsigned)m.len_v;
    if (limit > 0 && limit < total)  // only the set's first `limit` cells (rows of u)
        total = limit;
    float rs[K], rn[K], tn[K], sn[K], sf[K];
    size_t face[K];
    bool on[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const unsigned idx = idx0 + (unsigned)k * stride;
        on[k] = idx < total;
        const unsigned i = on[k] ? idx : 0u;
        const MurCellIdx c = mur_cell_idx(m, m.u0 + (int)(i % lu), m.v0 + (int)(i / lu), nx, ny, nz, pitch);
        face[k] = c.face;
        if (on[k]) {
            if constexpr (!UNI) {
                rs[k] = ms.slab[c.rs];
                rn[k] = ms.slab[c.rn];
            }
            tn[k] = ms.TN[c.nbr];
            sn[k] = ms.S[c.nbr];
            sf[k] = ms.S[c.face];
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (on[k]) {
            if constexpr (UNI)
                ms.T[face[k]] = mur_value_k(kf, tn[k], sn[k], sf[k]);
            else
                ms.T[face[k]] = mur_value(dt, ms.h, me, rs[k], rn[k], tn[k], sn[k], sf[k]);
        }
}

}  // namespace fdtd
