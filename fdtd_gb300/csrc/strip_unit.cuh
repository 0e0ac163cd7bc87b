// strip_unit.cuh -- device side of the compact forms' strip kernels (one
// work unit of the step), shared by the single-solve kernels
// (step_strip.cu) and the batched kernels (batch_strip.cu).
//
// Same update as the compact path of step_fused.cu (H, D increment and
// sources, Debye E and the recursion variable R, the x-face Mur updates),
// with the same arithmetic (cell_math.cuh, so both give the same bits), laid
// out to spend fewer instructions per cell:
//
// * A CTA of W warps owns a 32 x TY column tile (TY = RY * W) and a chunk of
//   z planes; lane l of warp w owns the strip of RY cells x0 + l, rows
//   y0 + w RY .. y0 + w RY + RY - 1.  Along the strip, the E^n rows read for
//   one cell's y + 1 neighbour are the next cell's own, and the D update
//   takes H^{n+1/2} at y - 1 from the previous cell of the strip, so only the
//   strip's first cell reads a row written by another warp.
// * Inputs arrive per plane by TMA tile loads into an S-deep mbarrier ring
//   (E^n with a one-cell halo, H^{n-1/2} with a low x / low y halo, the tile's
//   R, class bytes and, with 16-bit R, the rows' scale words).  Outputs go
//   the same way: each thread writes its results into dense shared-memory
//   tiles, over the boxes its plane was read from, and the plane's H^{n+1/2},
//   E^{n+1}, R^{n+1} (and scale words) leave by TMA stores.  No thread
//   computes a global address per cell.
// * A warp of its own moves the planes: it waits until the other warps have
//   consumed a plane, updates the x faces in its tiles, stores the tiles, waits
//   until the stores have read them and refills the stage.  With thread 0 of
//   the cell warps moving the planes, every plane of a CTA waited for its own
//   stores: 1.9 us per plane of a lone CTA against 1.4 (64^3, 32-bit R).
// * Tiles whose cells, halo included, all lie inside the update ranges of
//   every component, away from the x faces and from sources, take a path
//   without per-cell range tests (CTA-uniform choice, per plane for the
//   first and last planes of the grid); the other tiles take the tested
//   path.
//
// Cells the reference does not update get their old value in the stored tile
// (H^{n+1/2} = H^{n-1/2}; E^{n+1} = E^n, which equals the untouched slot's
// E^{n-1} because such cells are never written; R unchanged, or a zero
// residual with 16-bit R), so whole-tile stores leave them as the z-marching
// kernel leaves them.  The Mur kernel then updates the y and z faces.
#pragma once

#include "cell_math.cuh"
#include "native.cuh"
#include "tma_util.cuh"

namespace fdtd {
namespace strip {

using namespace tma;

constexpr int SX = 32;  // tile width in x: one warp's lanes

template <int RY, int W, bool R16>
struct StripGeo {
    static constexpr int TY = RY * W;
    static constexpr int CELL_THREADS = 32 * W, NTH = CELL_THREADS + 32;  // the cell warps, then the moving warp
    static_assert(TY % 4 == 0 && TY <= 32, "tile rows: a multiple of 4 (scale-word boxes) and one lane per row");
    static constexpr int EW = SX + 8, EH = TY + 2;  // E^n box: x0-4 .. x0+35, y0-1 .. y0+TY
    static constexpr int HW = SX + 4, HH = TY + 1;  // H box: x0-4 .. x0+31, y0-1 .. y0+TY-1
    static constexpr int RB = R16 ? 2 : 4;
    static constexpr int E_BYTES = EW * EH * 4, H_BYTES = HW * HH * 4, R_BYTES = SX * TY * RB, M_BYTES = SX * TY;
    static constexpr int X_BYTES = R16 ? TY * 4 : 0;
    // one ring stage
    static constexpr int OFF_E = 0;
    static constexpr int OFF_H = OFF_E + 3 * pad128(E_BYTES);
    static constexpr int OFF_R = OFF_H + 3 * pad128(H_BYTES);
    static constexpr int OFF_X = OFF_R + 3 * pad128(R_BYTES);
    static constexpr int OFF_M = OFF_X + pad128(X_BYTES);
    // x-face tiles: the Mur factors of the tile's rows ([TY] float4) of its
    // face (the near one when the tile holds both)
    static constexpr int F_BYTES = TY * 16;
    static constexpr int OFF_F = pad128(OFF_M + M_BYTES);
    static constexpr int STAGE = pad128(OFF_F + F_BYTES);
    static constexpr unsigned TX_FULL = 3u * E_BYTES + 3u * H_BYTES + 3u * R_BYTES + X_BYTES + M_BYTES;
    static constexpr unsigned TX_PRO = 3u * E_BYTES + 3u * H_BYTES;
    static constexpr unsigned TX_EPI = 3u * E_BYTES;
    // The output tiles (dense 32 x TY) live in the plane's own ring stage:
    // H^{n+1/2} and E^{n+1} over its E^n and H boxes (consumed by the H pass),
    // R^{n+1} and the scale words in place (each cell's by the thread that
    // read it).  They cost no shared memory; the stage's refill waits for its
    // stores to have read them.
    static constexpr int T_BYTES = SX * TY * 4;
    static constexpr int O_H = 0, O_E = 3 * T_BYTES;
    // and, in x-face tiles, E^n y, z of each face cell and of its x neighbour
    // ([face][TY] of ey, ez, neighbour's ey, ez) for the moving warp
    static constexpr int O_F = 6 * T_BYTES;
    static_assert(O_F + 2 * TY * 16 <= OFF_R, "the output tiles and the faces' E^n fit over the boxes");
    // H exchange of one plane: hz, hx of the row above each warp's first row
    // ([2][W][32]; row y0-1 for warp 0), and hz, hy of the x0-1 column
    // ([2][TY]).  Two sets, taken in turn by plane: a warp writes a plane's
    // set again two planes later, behind a barrier that every warp reaches
    // after reading it.
    static constexpr int XR = 2 * W * SX, XC = 2 * TY, XSET = XR + XC;
    // S barriers, then the give-up word
    template <int S>
    static constexpr int BAR_BYTES = (2 * S * 8 + 4 + 15) & ~15;
};

// Strip shapes: (cells per thread in y, warps per CTA).  0-2 use 8-row tiles
// (the same shared memory per CTA, 4, 8 or 2 warps), 3 uses 16-row tiles.
constexpr int STRIP_SHAPES = 4;
template <int SHAPE> struct Shape;
// BATCH_CTAS16 / BATCH_CTAS32: resident CTAs per SM the batched kernel is
// built for, with 16-bit and 32-bit R (its register bound; the solve's
// constants come from shared memory there).  Measured on the 64-solve batch:
// shape 0 with 16-bit R runs 2.6 % faster at 5 (no spills) than at 6 (80
// registers, spills), and with 32-bit R shared memory allows 5; shape 1
// spills 136-144 bytes at 5.
template <> struct Shape<0> { static constexpr int RY = 2, W = 4, BATCH_CTAS16 = 5, BATCH_CTAS32 = 5; };
template <> struct Shape<1> { static constexpr int RY = 1, W = 8, BATCH_CTAS16 = 4, BATCH_CTAS32 = 4; };
template <> struct Shape<2> { static constexpr int RY = 4, W = 2, BATCH_CTAS16 = 8, BATCH_CTAS32 = 8; };
template <> struct Shape<3> { static constexpr int RY = 4, W = 4, BATCH_CTAS16 = 2, BATCH_CTAS32 = 2; };

#ifndef FDTD_STRIP_STAGES
#define FDTD_STRIP_STAGES 3
#endif
constexpr int S_SEL = FDTD_STRIP_STAGES;  // ring stages

// Tensor maps of one strip launch over c's buffers for ty-row tiles (false:
// not TMA-addressable).
bool encode_strip_maps(const NativeConsts &c, bool r16, int ty, StripMaps *maps);

template <int RY, int W, int S, bool R16>
constexpr int strip_smem_bytes(int nclasses)
{
    using G = StripGeo<RY, W, R16>;
    return 128 + S * G::STAGE + 4 * 2 * G::XSET + G::template BAR_BYTES<S> + nclasses * 32;
}

struct StripArgs {
    NativeConsts c;
    int zchunk;
};



__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, uint32_t src, int x, int y, int z)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(x), "r"(y), "r"(z)
                 : "memory");
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// One thread arms the stage's barrier and issues the plane's boxes; no_r:
// the tile-plane holds no Debye memory, its R (and scale words) are not
// loaded.  With arm_only (the stall test hook) nothing is issued.
//
// A face tile's Mur factors: rows y0 .. of plane 0 of its x face (the near
// one when a tile of a grid at most 32 cells wide holds both; the far face's
// lanes then read theirs from global memory), nullptr in other tiles; plane z
// lies z * plane float4 further on.  bytes: the rows inside the grid x 16.
struct StripFaces {
    const float4 *src;
    size_t plane;
    uint32_t bytes;
};

template <int RY, int W, bool R16>
__device__ __forceinline__ void strip_issue(const StripMaps &maps, const StripFaces &f, unsigned char *stage,
                                            uint32_t bar, int kind, int x0, int y0, int z, bool arm_only, bool no_r)
{
    using G = StripGeo<RY, W, R16>;
    const unsigned full = (no_r ? G::TX_FULL - 3u * G::R_BYTES - G::X_BYTES : G::TX_FULL) + (f.src ? f.bytes : 0u);
    mbar_expect_tx(bar, kind == PLANE_FULL ? full : (kind == PLANE_PRO ? G::TX_PRO : G::TX_EPI));
    if (arm_only)
        return;
    for (int c = 0; c < 3; c++)
        tma_load_3d(smem_addr(stage + G::OFF_E + c * pad128(G::E_BYTES)), &maps.m[c], x0 - 4, y0 - 1, z, bar);
    if (kind == PLANE_EPI)
        return;
    for (int c = 0; c < 3; c++)
        tma_load_3d(smem_addr(stage + G::OFF_H + c * pad128(G::H_BYTES)), &maps.m[3 + c], x0 - 4, y0 - 1, z, bar);
    if (kind != PLANE_FULL)
        return;
    tma_load_3d(smem_addr(stage + G::OFF_M), &maps.m[9], x0, y0, z, bar);
    if (f.src)
        bulk_load(smem_addr(stage + G::OFF_F), f.src + (size_t)z * f.plane, f.bytes, bar);
    if (no_r)
        return;
    for (int c = 0; c < 3; c++)
        tma_load_3d(smem_addr(stage + G::OFF_R + c * pad128(G::R_BYTES)), &maps.m[6 + c], x0, y0, z, bar);
    if (R16)  // rows y0 .. y0+TY-1 of segment x0 / 32 (y0 * 4 bytes: 16-byte aligned)
        tma_load_3d(smem_addr(stage + G::OFF_X), &maps.m[10], y0, x0 / SX, z, bar);
}

// The constants the strip unit reads.  The single-solve kernel passes its
// NativeConsts parameter (constant bank); the batched kernel keeps this
// smaller copy of the current solve's in shared memory, with the source list
// left in the descriptor.
struct StripConsts {
    int nx, ny, nz;
    float kx, ky, kz, tx, ty, tz;
    int scheme, nsources;
    const int *sources;
    const DebyeCoef *coef;
    int nclasses;
    const float *jz;
    int njz;
    int step;
    int *step_counter;
    int *err;
    int fuse_mur_x;
    const float4 *mur_x;
};

__device__ __forceinline__ void strip_consts(StripConsts &o, const NativeConsts &c)
{
    o.nx = c.nx;
    o.ny = c.ny;
    o.nz = c.nz;
    o.kx = c.kx;
    o.ky = c.ky;
    o.kz = c.kz;
    o.tx = c.tx;
    o.ty = c.ty;
    o.tz = c.tz;
    o.scheme = c.scheme;
    o.nsources = c.nsources;
    o.sources = c.sources;
    o.coef = c.coef;
    o.nclasses = c.nclasses;
    o.jz = c.jz;
    o.njz = c.njz;
    o.step = c.step;
    o.step_counter = c.step_counter;
    o.err = c.err;
    o.fuse_mur_x = c.fuse_mur_x;
    o.mur_x = c.mur_x;
}

// Whether the columns x0..x0+31, rows y0..y0+ty-1, planes zc0..zc1-1 hold a source.
template <class C>
__device__ __forceinline__ bool strip_has_source(const C &c, int x0, int y0, int ty, int zc0, int zc1)
{
    bool any = false;
    for (int s = 0; s < c.nsources; s++) {
        const int sx = c.sources[3 * s], sy = c.sources[3 * s + 1], sz = c.sources[3 * s + 2];
        any |= sx >= x0 && sx < x0 + SX && sy >= y0 && sy < y0 + ty && sz >= zc0 && sz < zc1;
    }
    return any;
}

// A CTA's shared memory: S ring stages, the two H exchange sets, the S
// barriers, the give-up word, the class table.
struct StripSmem {
    unsigned char *stages;
    float *xch;
    uint64_t *full, *consumed;
    int *stop;
    DebyeCoef *coef;
};

template <int RY, int W, int S, bool R16>
__device__ __forceinline__ StripSmem strip_smem(unsigned char *smem_raw)
{
    using G = StripGeo<RY, W, R16>;
    StripSmem m;
    m.stages = smem_raw + ((128 - (smem_addr(smem_raw) & 127)) & 127);
    m.xch = reinterpret_cast<float *>(m.stages + S * G::STAGE);
    m.full = reinterpret_cast<uint64_t *>(m.xch + 2 * G::XSET);
    m.consumed = m.full + S;
    m.stop = reinterpret_cast<int *>(m.consumed + S);
    m.coef = reinterpret_cast<DebyeCoef *>(reinterpret_cast<unsigned char *>(m.full) + G::template BAR_BYTES<S>);
    return m;
}

template <int W, int S>
__device__ __forceinline__ void strip_init_bars(const StripSmem &m)
{
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(smem_addr(&m.full[s]), 1);
            mbar_init(smem_addr(&m.consumed[s]), W);
        }
        *m.stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

template <class C>
__device__ __forceinline__ void strip_load_coef(const C &c, DebyeCoef *coef, int nthreads)
{
    const float *src = reinterpret_cast<const float *>(c.coef);
    float *dst = reinterpret_cast<float *>(coef);
    for (int i = threadIdx.x; i < c.nclasses * 8; i += nthreads)
        dst[i] = src[i];
}

// The planes of a unit as the moving warp and the cell warps see them: the
// unit's first plane p0, its planes (prologue and epilogue included) and the
// ring's stages and barrier phases.
template <int RY, int W, int S, bool R16>
struct StripPlanes {
    using G = StripGeo<RY, W, R16>;
    const StripSmem &sm;
    int zc0, zc1, p0, nplanes;
    unsigned long long memless;  // bit j: plane zc0 + j of the tile holds no Debye memory
    __device__ __forceinline__ StripPlanes(const StripSmem &m, int nz, int zchunk, int bz, unsigned long long ml)
        : sm(m), zc0(bz * zchunk), zc1(min(nz, bz * zchunk + zchunk)), p0(max(zc0 - 1, 0)),
          nplanes(min(zc1, nz - 1) - p0 + 1), memless(ml)
    {
    }
    __device__ __forceinline__ unsigned char *stage(int k) const { return sm.stages + (k % S) * G::STAGE; }
    __device__ __forceinline__ uint32_t full(int k) const { return smem_addr(&sm.full[k % S]); }
    __device__ __forceinline__ uint32_t consumed(int k) const { return smem_addr(&sm.consumed[k % S]); }
    __device__ __forceinline__ uint32_t parity(int k) const { return (uint32_t)((k / S) & 1); }
    __device__ __forceinline__ bool no_r(int z) const { return z >= zc0 && ((memless >> (z - zc0)) & 1ull) != 0; }
};

// The moving warp's copies: a plane's boxes into its stage, a plane's tiles
// from it.
template <int RY, int W, int S, bool R16>
struct StripMove {
    using G = StripGeo<RY, W, R16>;
    const StripMaps &maps;
    const StripPlanes<RY, W, S, R16> &u;
    StripFaces faces;
    int x0, y0;
    __device__ __forceinline__ void issue(int k, bool arm_only) const
    {
        const int z = u.p0 + k;
        strip_issue<RY, W, R16>(maps, faces, u.stage(k), u.full(k), plane_kind(z, u.zc0, u.zc1), x0, y0, z, arm_only,
                                u.no_r(z));
    }
    __device__ __forceinline__ void store(int k) const
    {
        const int z = u.p0 + k;
        const uint32_t ob = smem_addr(u.stage(k));
        const bool no_r = u.no_r(z);
        for (int comp = 0; comp < 3; comp++) {
            tma_store_3d(&maps.m[11 + comp], ob + G::O_H + comp * G::T_BYTES, x0, y0, z);
            tma_store_3d(&maps.m[14 + comp], ob + G::O_E + comp * G::T_BYTES, x0, y0, z);
            if (!no_r)
                tma_store_3d(&maps.m[6 + comp], ob + G::OFF_R + comp * pad128(G::R_BYTES), x0, y0, z);
        }
        if (R16 && !no_r)
            tma_store_3d(&maps.m[10], ob + G::OFF_X, y0, x0 / SX, z);
        bulk_commit();
    }
};

// The x faces of a unit: the moving warp applies their Mur updates to a
// plane's E tiles before it stores them (updateMurBoundary ey/ez x faces,
// fdtd_calculations.cu:280-340; the same rounded operations as the Mur
// kernel).  Lane row + TY * face (0 near, 1 far) updates one face cell from the
// neighbour's E^{n+1} in the tile and the E^n that the cell warps left beside
// it.  In the cell warps these updates cost four shuffles, two more loads and
// a divergent branch per row in every warp of a face tile.  us per step with
// them there (and the moving warp's lane 0 at work alone) and so, 16-bit R: 20
// solves of 48-256 cells per axis 437 and 411, of 24-128 109 and 99; 301 x 245 x
// 187 154 and 143, 150 x 134 x 170 47.8 and 44.2, 512 x 512 x 400 922 and 907;
// 32-bit R: 431 and 418, 152 and 149, 48.6 and 47.0, 992 and 994.
struct StripXFaces {
    const float4 *mur_x;  // Mur factors, [face][z][y]
    int nx, ny, nz, scheme;
    bool near, far;       // the tile holds x = 0, x = nx - 1
};

template <int RY, int W, int S, bool R16>
__device__ __forceinline__ void strip_mur_rows(const StripMove<RY, W, S, R16> &move, const StripXFaces &f, int k, int lane)
{
    using G = StripGeo<RY, W, R16>;
    constexpr int TY = G::TY, TS = SX * TY;
    static_assert(2 * TY <= 32, "a lane per row of either face");
    const int z = move.u.p0 + k, face = lane / TY, row = lane % TY, y = move.y0 + row;
    if (z < 1 || z >= f.nz - 1 || face > 1 || !(face ? f.far : f.near) || y > f.ny - 2)
        return;
    unsigned char *stage = move.u.stage(k);
    float *ey = reinterpret_cast<float *>(stage + G::O_E) + TS + row * SX, *ez = ey + TS;
    const float4 e0 = reinterpret_cast<const float4 *>(stage + G::O_F)[face * TY + row];
    const float4 mf = face && f.near ? f.mur_x[((size_t)f.nz + z) * f.ny + y]
                                     : reinterpret_cast<const float4 *>(stage + G::OFF_F)[row];
    const int self = face ? f.nx - 1 - move.x0 : 0, nbr = face ? self - 1 : 1;
    auto mur = [&](float tn, float sn, float sf) {
        return __fmul_rn(mf.x, __fsub_rn(__fadd_rn(__fmul_rn(mf.y, tn), __fmul_rn(mf.z, sn)), __fmul_rn(mf.w, sf)));
    };
    // ey: y 0..ny-2, z 1..nz-2; fdtd_calculations.cu:323: the far ey face
    // reads E^n at x-1 in both terms
    ey[self] = mur(face && f.scheme != FDTD_SCHEME_CORRECTED ? e0.z : ey[nbr], e0.z, e0.x);
    if (y >= 1)  // ez: y 1..ny-2 (z = 0 in the Mur kernel)
        ez[self] = mur(ez[nbr], e0.w, e0.y);
}

// The moving warp at work: fills the ring, then plane by plane waits until the
// cell warps have consumed the plane, applies the x-face Mur updates, stores
// the tiles the cell warps have left in its stage and refills the stage; all
// but the updates by one elected lane.  Its waits are bounded; when one gives
// up, or a cell warp's did (the stop word), the error flag is raised (where only
// stores are left the cell warps miss nothing, and the tiles would be lost in
// silence), the copies in flight land (bounded) and the unit ends.  stall: test
// hook (STALL_*).
//
// A plane's refill waits for this warp, so its own instructions count.  The
// warp stays together, its lane chosen by elect.sync (the compiler then keeps
// the copies' operands in uniform registers; lane == 0 with a shuffle 1011 us
// where this takes 994, the other lanes gone 1031), and the issuing code is
// there once (the kernel's loops compete for the instruction cache: 930 us
// with the first fill apart, 920 so; 512 x 512 x 400, 32-bit R and 16-bit R).
template <int RY, int W, int S, bool R16>
__device__ __forceinline__ void strip_run(const StripMove<RY, W, S, R16> &move, const StripXFaces &f, int *err,
                                          int lane, int stall)
{
    const auto &u = move.u;
    const bool one = elect_one();
    stall = __shfl_sync(0xffffffffu, stall, 0);  // lane 0 was told
    const int end = stall == STALL_STORE ? u.zc1 - 1 : u.zc1;
    // the ring's first fill is the loop's first S turns
    int k = -S;
    for (; u.p0 + k < end; k++) {
        if (k >= 0) {
            bool ok = false;
            if (one)
                ok = mbar_wait(u.consumed(k), u.parity(k)) && !*static_cast<volatile int *>(u.sm.stop);
            if (!__any_sync(0xffffffffu, ok))
                break;
            const bool out = u.p0 + k >= u.zc0;
            if (out && (f.near || f.far)) {
                __syncwarp();  // every lane sees what the waiting lane was given
                strip_mur_rows(move, f, k, lane);
                fence_async_shared();  // the lanes' writes are visible to the stores
                __syncwarp();
            }
            if (one && out)
                move.store(k);
        }
        if (one && k + S < u.nplanes) {
            bulk_wait_read<0>();  // the refill overwrites the tiles
            move.issue(k + S, stall == STALL_LOAD && k + S == 1);
        }
    }
    if (one && u.p0 + k < u.zc1) {  // a wait gave up
        atomicExch(err, 1);
        for (int j = k; j < u.nplanes && j < k + S; j++)
            mbar_wait(u.full(j), u.parity(j));
    }
    if (one)
        bulk_wait_all();
}

// One work unit: column tile (bx, by), z chunk bz of one solve.  memless: bit
// j set when plane zc0 + j of the tile holds no Debye memory.  stall: the
// test hook of strip_run.  When a bounded wait gives up the error flag is
// raised and the unit ends.
template <int RY, int W, int S, bool R16, class C>
__device__ __forceinline__ void strip_unit(const C &c, const StripMaps &maps, int zchunk, int bx, int by,
                                           int bz, unsigned long long memless, const StripSmem &sm, int stall)
{
    using G = StripGeo<RY, W, R16>;
    constexpr int TY = G::TY;
    const int nx = c.nx, ny = c.ny, nz = c.nz;
    const int tid = threadIdx.x, lane = tid & 31;
    // by a shuffle: the compiler then knows the warp index as uniform over the
    // warp, and keeps the plane loop's addresses in uniform registers behind the
    // moving warp's branch (without it the 16-bit form ran 6 % slower)
    const int w = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int x0 = bx * SX, y0 = by * TY;
    const StripPlanes<RY, W, S, R16> u(sm, nz, zchunk, bz, memless);
    const int zc0 = u.zc0, zc1 = u.zc1, p0 = u.p0, nplanes = u.nplanes;

    // x-face Mur updates in the tiles that hold x = 0 or nx-1, by the moving
    // warp; their per-cell factors arrive with the plane's boxes
    const int mur_bits = mur_x_fused_faces(c);
    const bool face_near = (mur_bits & 1) && x0 == 0;
    const bool face_far_cta = (mur_bits & 2) && x0 <= nx - 1 && nx - 1 < x0 + SX;
    const bool face_cta = face_near || face_far_cta;
    if (w == W) {
        StripMove<RY, W, S, R16> move{maps, u, StripFaces{nullptr, (size_t)ny, 0u}, x0, y0};
        if (face_cta) {
            move.faces.bytes = (uint32_t)min(TY, ny - y0) * 16u;
            move.faces.src = face_near ? c.mur_x + y0 : c.mur_x + (size_t)nz * ny + y0;
        }
        strip_run(move, StripXFaces{c.mur_x, nx, ny, nz, c.scheme, face_near, face_far_cta}, c.err, lane, stall);
        return;
    }

    const DebyeCoef *coef = sm.coef;
    const int x = x0 + lane, ry0 = w * RY;  // first row of this thread's strip, relative to y0
    const bool unit_src = strip_has_source(c, x0, y0, TY, zc0, zc1);
    float jz_now = 0.0f;
    if (unit_src) {
        const int n = c.step_counter ? *c.step_counter : c.step;
        const int j = c.scheme == FDTD_SCHEME_CORRECTED ? n : n - n % 3;
        jz_now = (j >= 0 && j < c.njz) ? c.jz[j] : 0.0f;
    }
    const float kx = c.kx, ky = c.ky, kz = c.kz, tcx = c.tx, tcy = c.ty, tcz = c.tz;
    const int cls_max = c.nclasses - 1;
    // every own cell and every halo cell inside the update ranges of all
    // components in x and y, no x face, no source
    const bool xy_inside = x0 >= 1 && x0 + SX - 1 <= nx - 2 && y0 >= 1 && y0 + TY - 1 <= ny - 2 && !face_cta &&
                           !unit_src;

    // Range-tested tiles: each component's update range in x and y per row
    // of the strip (fixed for the unit; the z ranges are per plane).  The
    // tested path computes every update and keeps it where its range holds.
    enum : unsigned { M_HX = 1, M_HY = 2, M_HZ = 4, M_E0 = 8, M_E1 = 16, M_E2 = 32, M_EYZ = 64, M_DOM = 128 };
    unsigned mrow = 0;  // 8 bits per row of the strip
#pragma unroll
    for (int r = 0; r < RY; r++) {
        const int y = y0 + ry0 + r;
        const bool in_dom = x < nx && y < ny;
        const bool xi = x >= 1 && x < nx - 1, yi = y >= 1 && y < ny - 1;
        unsigned m = 0;
        m |= (xi && y < ny - 1) ? M_HX : 0u;
        m |= (x < nx - 1 && yi) ? M_HY : 0u;
        m |= (x < nx - 1 && y < ny - 1) ? M_HZ : 0u;
        m |= (in_dom && x < nx - 1 && yi) ? M_E0 : 0u;
        m |= (in_dom && xi && y < ny - 1) ? M_E1 : 0u;
        m |= (in_dom && xi && yi) ? M_E2 : 0u;
        m |= (in_dom && x >= 1) ? M_EYZ : 0u;
        m |= in_dom ? M_DOM : 0u;
        mrow |= m << (8 * r);
    }
    auto has = [&](int r, unsigned bit) { return ((mrow >> (8 * r)) & bit) != 0u; };

    float hxm[RY], hym[RY];  // H^{n+1/2} x, y of the strip's cells at z-1
#pragma unroll
    for (int r = 0; r < RY; r++)
        hxm[r] = hym[r] = 0.0f;

    // this warp is done with the plane in ring stage `slot` (its writes to the
    // stage are visible to the TMA stores)
    auto consumed = [&](int slot) {
        fence_async_shared();
        __syncwarp();
        if (lane == 0)
            mbar_arrive(smem_addr(&sm.consumed[slot]));
    };
    auto give_up = [&](int slot) {
        if (tid == 0) {
            atomicExch(c.err, 1);
            *static_cast<volatile int *>(sm.stop) = 1;
        }
        consumed(slot);
    };
    int slot = 0, next = 1;   // ring stages of planes k and k + 1 (S > 1)
    uint32_t phase_next = 0;  // barrier phase of plane k + 1
    for (int k = 0; p0 + k < zc1; k++, slot = next, next = next + 1 == S ? 0 : next + 1, phase_next ^= next == 0) {
        const int z = p0 + k;
        bool ok = true;
        if (k == 0)
            ok = mbar_wait(smem_addr(&sm.full[0]), 0);
        if (ok && k + 1 < nplanes)
            ok = mbar_wait(smem_addr(&sm.full[next]), phase_next);
        unsigned char *stage = sm.stages + slot * G::STAGE;
        const float *EA = reinterpret_cast<const float *>(stage + G::OFF_E);
        const float *EB = reinterpret_cast<const float *>(sm.stages + next * G::STAGE + G::OFF_E);
        const float *HA = reinterpret_cast<const float *>(stage + G::OFF_H);
        // this plane's H exchange set
        float *xr = sm.xch + (k & 1) * G::XSET, *xc = xr + G::XR;
        constexpr int ES = pad128(G::E_BYTES) / 4, HS = pad128(G::H_BYTES) / 4;
        auto ea = [&](int comp, int r, int cc) { return EA[comp * ES + r * G::EW + cc]; };
        auto eb = [&](int comp, int r, int cc) { return EB[comp * ES + r * G::EW + cc]; };
        auto ha = [&](int comp, int r, int cc) { return HA[comp * HS + r * G::HW + cc]; };
        const bool zlo = z < nz - 1, zmid = z >= 1 && z < nz - 1;
        const bool fast = xy_inside && zmid;  // uniform over the CTA
        const int ec = lane + 4;

        // ---- H^{n+1/2} at plane z on the strip (fdtd_calculations.cu:43-76)
        float ex[RY + 1], ey[RY], ez[RY + 1];
        float hxn[RY], hyn[RY], hzn[RY];
#pragma unroll
        for (int r = 0; r <= RY; r++) {
            ex[r] = ea(0, ry0 + r + 1, ec);
            ez[r] = ea(2, ry0 + r + 1, ec);
        }
#pragma unroll
        for (int r = 0; r < RY; r++) {
            const int er = ry0 + r + 1;
            ey[r] = ea(1, er, ec);
            hxn[r] = ha(0, er, ec);
            hyn[r] = ha(1, er, ec);
            hzn[r] = ha(2, er, ec);
            if (fast) {
                hxn[r] = cm_h(hxn[r], ky, ez[r + 1], ez[r], ky, eb(1, er, ec), ey[r]);
                hyn[r] = cm_h(hyn[r], kz, eb(0, er, ec), ex[r], kx, ea(2, er, ec + 1), ez[r]);
                hzn[r] = cm_h(hzn[r], kx, ea(1, er, ec + 1), ey[r], ky, ex[r + 1], ex[r]);
            } else {
                const float vx = cm_h(hxn[r], ky, ez[r + 1], ez[r], ky, eb(1, er, ec), ey[r]);
                const float vy = cm_h(hyn[r], kz, eb(0, er, ec), ex[r], kx, ea(2, er, ec + 1), ez[r]);
                const float vz = cm_h(hzn[r], kx, ea(1, er, ec + 1), ey[r], ky, ex[r + 1], ex[r]);
                hxn[r] = has(r, M_HX) && zlo ? vx : hxn[r];
                hyn[r] = has(r, M_HY) && zlo ? vy : hyn[r];
                hzn[r] = has(r, M_HZ) && zmid ? vz : hzn[r];
            }
        }
        if (z < zc0) {  // chunk prologue: only the strip's H x, y at zc0 - 1 are needed
#pragma unroll
            for (int r = 0; r < RY; r++) {
                hxm[r] = hxn[r];
                hym[r] = hyn[r];
            }
            if (cells_barrier_or<G::CELL_THREADS>(!ok)) {
                give_up(slot);
                return;
            }
            consumed(slot);
        } else {
            if (w + 1 < W) {
                xr[(w + 1) * SX + lane] = hzn[RY - 1];
                xr[(W + w + 1) * SX + lane] = hxn[RY - 1];
            }
            if (w == 0) {  // row y0 - 1: hx, hz (box row 0)
                const float ex_ = ea(0, 0, ec), ey_ = ea(1, 0, ec), ez_ = ea(2, 0, ec);
                float vx = ha(0, 0, ec), vz = ha(2, 0, ec);
                if (fast) {
                    vx = cm_h(vx, ky, ez[0], ez_, ky, eb(1, 0, ec), ey_);
                    vz = cm_h(vz, kx, ea(1, 0, ec + 1), ey_, ky, ex[0], ex_);
                } else if (y0 >= 1 && x < nx) {
                    if (x >= 1 && x < nx - 1 && zlo)
                        vx = cm_h(vx, ky, ez[0], ez_, ky, eb(1, 0, ec), ey_);
                    if (x < nx - 1 && zmid)
                        vz = cm_h(vz, kx, ea(1, 0, ec + 1), ey_, ky, ex[0], ex_);
                } else {
                    vx = vz = 0.0f;
                }
                xr[lane] = vz;
                xr[W * SX + lane] = vx;
            }
            if (w == W - 1 && lane < TY) {  // column x0 - 1: hy, hz of row y0 + lane (box column 3)
                const int er = lane + 1, cc = 3, yy = y0 + lane;
                const float ex_ = ea(0, er, cc), ey_ = ea(1, er, cc), ez_ = ea(2, er, cc);
                float vy = ha(1, er, cc), vz = ha(2, er, cc);
                if (fast) {
                    vy = cm_h(vy, kz, eb(0, er, cc), ex_, kx, ea(2, er, cc + 1), ez_);
                    vz = cm_h(vz, kx, ea(1, er, cc + 1), ey_, ky, ea(0, er + 1, cc), ex_);
                } else if (x0 >= 1 && yy < ny) {
                    if (yy >= 1 && yy < ny - 1 && zlo)
                        vy = cm_h(vy, kz, eb(0, er, cc), ex_, kx, ea(2, er, cc + 1), ez_);
                    if (x0 - 1 < nx - 1 && yy < ny - 1 && zmid)
                        vz = cm_h(vz, kx, ea(1, er, cc + 1), ey_, ky, ea(0, er + 1, cc), ex_);
                } else {
                    vy = vz = 0.0f;
                }
                xc[lane] = vz;
                xc[TY + lane] = vy;
            }
            // the cell warps decide here whether a wait gave up (nothing has
            // reached global memory from this plane yet)
            if (cells_barrier_or<G::CELL_THREADS>(!ok)) {
                give_up(slot);
                return;
            }

            // ---- D increment, sources, E^{n+1} and R^{n+1} on the strip
            const bool plane_no_r = u.no_r(z);  // uniform: R is +0 on every cell of the tile-plane
            float *OH = reinterpret_cast<float *>(stage + G::O_H);
            float *OE = reinterpret_cast<float *>(stage + G::O_E);
            const unsigned char *M = stage + G::OFF_M;
            constexpr int TS = SX * TY;  // elements of one dense tile
            // every operand of the strip first, every result last: the stores may
            // alias the loads, so the compiler keeps their order
            float hz_xm[RY], hy_xm[RY], r0[RY], r1[RY], r2[RY];
            DebyeCoef kcs[RY];
            const float hz_row = xr[w * SX + lane], hx_row = xr[(W + w) * SX + lane];
#pragma unroll
            for (int r = 0; r < RY; r++) {
                const int row = ry0 + r, t = row * SX + lane;
                const float hz_up = __shfl_up_sync(0xffffffffu, hzn[r], 1);
                const float hy_up = __shfl_up_sync(0xffffffffu, hyn[r], 1);
                hz_xm[r] = lane ? hz_up : xc[row];
                hy_xm[r] = lane ? hy_up : xc[TY + row];
                kcs[r] = coef[min((int)M[t], cls_max)];
                if (plane_no_r) {
                    r0[r] = r1[r] = r2[r] = 0.0f;
                } else if constexpr (R16) {
                    const unsigned short *RT = reinterpret_cast<const unsigned short *>(stage + G::OFF_R);
                    constexpr int RS = pad128(G::R_BYTES) / 2;
                    const float sc = cm_r16_scale(reinterpret_cast<const uint32_t *>(stage + G::OFF_X)[row]);
                    r0[r] = cm_r16_r(RT[t], sc, kcs[r].a, ex[r]);
                    r1[r] = cm_r16_r(RT[RS + t], sc, kcs[r].a, ey[r]);
                    r2[r] = cm_r16_r(RT[2 * RS + t], sc, kcs[r].a, ez[r]);
                } else {
                    const float *RT = reinterpret_cast<const float *>(stage + G::OFF_R);
                    constexpr int RS = pad128(G::R_BYTES) / 4;
                    r0[r] = RT[t];
                    r1[r] = RT[RS + t];
                    r2[r] = RT[2 * RS + t];
                }
            }
            float en[3][RY], rn[3][RY];
#pragma unroll
            for (int r = 0; r < RY; r++) {
                const int row = ry0 + r, y = y0 + row;
                const float hz_ym = r ? hzn[r - 1] : hz_row;
                const float hx_ym = r ? hxn[r - 1] : hx_row;
                const DebyeCoef &kc = kcs[r];
                const float k12 = cm_k12(kc);
                float en0, en1, en2, rn0, rn1, rn2;
                if (fast) {
                    const float g0 = cm_dinc(tcy, hzn[r], hz_ym, tcz, hyn[r], hym[r]);
                    const float g1 = cm_dinc(tcz, hxn[r], hxm[r], tcx, hzn[r], hz_xm[r]);
                    const float g2 = cm_dinc(tcx, hyn[r], hy_xm[r], tcy, hxn[r], hx_ym);
                    en0 = cm_e_next(kc, k12, ex[r], g0, r0[r]);
                    en1 = cm_e_next(kc, k12, ey[r], g1, r1[r]);
                    en2 = cm_e_next(kc, k12, ez[r], g2, r2[r]);
                    rn0 = cm_r_next(kc, ex[r], g0);
                    rn1 = cm_r_next(kc, ey[r], g1);
                    rn2 = cm_r_next(kc, ez[r], g2);
                    if constexpr (R16) {
                        rn0 = cm_r16_rho(kc.a, en0, rn0);
                        rn1 = cm_r16_rho(kc.a, en1, rn1);
                        rn2 = cm_r16_rho(kc.a, en2, rn2);
                    }
                } else {
                    const bool ex_on = has(r, M_E0) && zmid;  // also the range of g0
                    const float g0 = ex_on ? cm_dinc(tcy, hzn[r], hz_ym, tcz, hyn[r], hym[r]) : 0.0f;
                    const float g1 =
                        has(r, M_E1) && zmid ? cm_dinc(tcz, hxn[r], hxm[r], tcx, hzn[r], hz_xm[r]) : 0.0f;
                    bool src = false;
                    if (unit_src)
                        for (int s = 0; s < c.nsources; s++)
                            src |= c.sources[3 * s + 2] == z && c.sources[3 * s] == x && c.sources[3 * s + 1] == y;
                    const float d2 = cm_dinc(tcx, hyn[r], hy_xm[r], tcy, hxn[r], hx_ym);
                    const float g2 = has(r, M_DOM) && ((has(r, M_E2) && zlo) || src)
                                         ? (src ? __fsub_rn(d2, jz_now) : d2)
                                         : 0.0f;
                    const bool eyz_on = has(r, M_EYZ) && z >= 1;
                    // not updated: E keeps E^n, R keeps R^n (16-bit R: residual 0)
                    const float u0 = cm_e_next(kc, k12, ex[r], g0, r0[r]);
                    const float u1 = cm_e_next(kc, k12, ey[r], g1, r1[r]);
                    const float u2 = cm_e_next(kc, k12, ez[r], g2, r2[r]);
                    float s0 = cm_r_next(kc, ex[r], g0), s1 = cm_r_next(kc, ey[r], g1), s2 = cm_r_next(kc, ez[r], g2);
                    if constexpr (R16) {
                        s0 = cm_r16_rho(kc.a, u0, s0);
                        s1 = cm_r16_rho(kc.a, u1, s1);
                        s2 = cm_r16_rho(kc.a, u2, s2);
                    }
                    en0 = ex_on ? u0 : ex[r];
                    en1 = eyz_on ? u1 : ey[r];
                    en2 = eyz_on ? u2 : ez[r];
                    rn0 = ex_on ? s0 : (R16 ? 0.0f : r0[r]);
                    rn1 = eyz_on ? s1 : (R16 ? 0.0f : r1[r]);
                    rn2 = eyz_on ? s2 : (R16 ? 0.0f : r2[r]);
                }
                en[0][r] = en0;
                en[1][r] = en1;
                en[2][r] = en2;
                rn[0][r] = rn0;
                rn[1][r] = rn1;
                rn[2][r] = rn2;
            }
#pragma unroll
            for (int r = 0; r < RY; r++) {
                const int row = ry0 + r, t = row * SX + lane, y = y0 + row;
                if (face_cta) {  // E^n of the face cells and their neighbours, for the moving warp
                    float2 *EF = reinterpret_cast<float2 *>(stage + G::O_F);
                    const int to_far = nx - 1 - x;  // 0: the far face cell, 1: its neighbour
                    if (face_near && lane < 2)
                        EF[2 * row + lane] = make_float2(ey[r], ez[r]);
                    if (face_far_cta && (to_far == 0 || to_far == 1))
                        EF[2 * (TY + row) + to_far] = make_float2(ey[r], ez[r]);
                }
                OH[t] = hxn[r];
                OH[TS + t] = hyn[r];
                OH[2 * TS + t] = hzn[r];
                OE[t] = en[0][r];
                OE[TS + t] = en[1][r];
                OE[2 * TS + t] = en[2][r];
                if (plane_no_r) {
                    // R stays +0: nothing to store
                } else if constexpr (R16) {
                    // one warp is one row segment: every cell of it is
                    // rewritten with the segment's new scale
                    unsigned short h0, h1, h2;
                    const uint32_t b = cm_r16_encode(rn[0][r], rn[1][r], rn[2][r], h0, h1, h2);
                    unsigned short *OR = reinterpret_cast<unsigned short *>(stage + G::OFF_R);
                    constexpr int RS = pad128(G::R_BYTES) / 2;
                    OR[t] = h0;
                    OR[RS + t] = h1;
                    OR[2 * RS + t] = h2;
                    if (lane == 0)
                        reinterpret_cast<uint32_t *>(stage + G::OFF_X)[row] = y < ny ? b : 0u;
                } else {
                    float *OR = reinterpret_cast<float *>(stage + G::OFF_R);
                    constexpr int RS = pad128(G::R_BYTES) / 4;
                    OR[t] = rn[0][r];
                    OR[RS + t] = rn[1][r];
                    OR[2 * RS + t] = rn[2][r];
                }
                hxm[r] = hxn[r];
                hym[r] = hyn[r];
            }
            consumed(slot);
        }
    }
}

}  // namespace strip
}  // namespace fdtd
