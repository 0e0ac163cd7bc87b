// compat.cu -- reference-compatible launchers (fdtd_calculations.h:18-42).
//
// Same argument lists and per-component index ranges as the reference's five
// kernels, over the reference's float material arrays and three-slot state.
// The grids differ: thread tiles (of several z planes for H and D) instead of
// 128 x 1 rows, sources as one warp instead of a full grid, Mur over
// the face cells only.  The kernels are programmatic dependents of the stream's
// previous launch: one after another on a small grid they took 4.2-5.4 us each,
// so 2.7-4.
#include <algorithm>
#include <array>
#include <atomic>

#include "device_common.cuh"

namespace fdtd {
namespace {

// The reference's __constant__ block (fdtd_calculations.h:10-15).
struct SymbolBlock {
    int nx, ny, nz;
    float dt, dx, dy, dz, mu0, eps0;
    int nsources;
    int sources[3 * FDTD_MAX_SOURCES];
    int njz;
};

__constant__ SymbolBlock c_sym;
// The whole source table; the reference's dJz holds 512 entries.
__device__ float g_jz[FDTD_JZ_LEN];

std::array<std::atomic<bool>, 128> g_symbols_ready{};
std::array<SymbolBlock, 128> g_host_sym{};

int current_device_checked(int *dev)
{
    cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess)
        return e;
    if (*dev < 0 || *dev >= (int)g_symbols_ready.size())
        return FDTD_ERR_INVALID;
    return FDTD_OK;
}

// Thread tile: long rows share their 32-byte sectors and E and H neighbours within
// a block (five launchers on 256 x 256 x 200: 343 us with 32 x 8, 338 with 64 x 2, 335
// with 256 x 1).  Narrow grids take the power of two that holds a row, so that no
// more than half of the threads idle: E kernel on 8 x 600 x 600 182 us in 64 x 2
// tiles, 43 so (32 x 8: 115), 16 x 512 x 512 133 and 58 (95), 32 x 512 x 256 68 and
// 57 (64).
constexpr int TILE_THREADS = 128;

dim3 cell_tile(int nx)
{
    const int tx = nx <= 8 ? 8 : nx <= 16 ? 16 : nx <= 32 ? 32 : 64;
    return dim3(tx, TILE_THREADS / tx);
}

// z planes per thread of the H and D kernels, bound by HBM (36 bytes per cell).
// With one plane per thread, each component loaded, updated and stored in
// turn, they ran 114 and 117 us on 256 x 256 x 200 (4.1 and 4.0 TB/s): few loads
// in flight, and E or H of the neighbouring plane read again through L2.  With
// all loads first and 1 / 2 / 4 / 8 planes per thread: H 83 / 81 / 79 / 84 us, D 86
// / 83 / 82 / 90.
constexpr int H_PLANES = 4, D_PLANES = 4;

__global__ void __launch_bounds__(TILE_THREADS) compat_h_kernel(float *hx, float *hy,
                                                         float *hz, const float *ex,
                                                         const float *ey, const float *ez)
{
    pdl_begin();
    const int nx = c_sym.nx, ny = c_sym.ny, nz = c_sym.nz;
    const TileXY t(nx, blockDim.x, blockDim.y);
    const int x = t.x0 + threadIdx.x, y = t.y0 + threadIdx.y;
    if (x >= nx - 1 || y >= ny - 1)
        return;
    const float dt = c_sym.dt, mu0 = c_sym.mu0;
    const float kx = dt / (mu0 * c_sym.dx), ky = dt / (mu0 * c_sym.dy), kz = dt / (mu0 * c_sym.dz);
    const float *const in[3] = {hx, hy, hz};
    float *const out[3] = {hx, hy, hz};
    h_column<H_PLANES>(x, y, blockIdx.y * H_PLANES, nx, ny, nz, nx, kx, ky, kz, ex, ey, ez, in, out);
}

__global__ void __launch_bounds__(TILE_THREADS) compat_d_kernel(float *dxT, float *dyT,
                                                         float *dzT, const float *dxS,
                                                         const float *dyS, const float *dzS,
                                                         const float *hx, const float *hy,
                                                         const float *hz)
{
    pdl_begin();
    constexpr int K = D_PLANES;
    const int nx = c_sym.nx, ny = c_sym.ny, nz = c_sym.nz;
    const TileXY t(nx, blockDim.x, blockDim.y);
    const int x = t.x0 + threadIdx.x, y = t.y0 + threadIdx.y, z0 = blockIdx.y * K;
    if (x >= nx - 1 || y >= ny - 1)
        return;  // no D component is updated at x = nx-1, y = ny-1 or z = nz-1
    const int n = min(K, nz - 1 - z0);
    const float tx = c_sym.dt / c_sym.dx, ty = c_sym.dt / c_sym.dy, tz = c_sym.dt / c_sym.dz;
    const size_t i = cell_index(x, y, z0, nx, ny), sy = nx, sz = (size_t)nx * ny;
    const bool xi = x >= 1, yi = y >= 1;
    // every load before the first store; H x, y of a plane are read once for
    // the cells above and below it
    float a[K + 1], b[K + 1], c[K], ay[K], bx[K], cx[K], cy[K], d[3][K];
    a[0] = b[0] = 0.0f;
    if (z0 >= 1) {
        a[0] = hx[i - sz];
        b[0] = hy[i - sz];
    }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (k < n) {
            const size_t j = i + k * sz;
            a[k + 1] = hx[j];
            b[k + 1] = hy[j];
            c[k] = hz[j];
            if (yi) {
                ay[k] = hx[j - sy];
                cy[k] = hz[j - sy];
                d[0][k] = dxS[j];
            }
            if (xi) {
                bx[k] = hy[j - 1];
                cx[k] = hz[j - 1];
                d[1][k] = dyS[j];
            }
            if (xi && yi)
                d[2][k] = dzS[j];
        }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (k < n) {
            const size_t j = i + k * sz;
            const bool zi = z0 + k >= 1;
            if (yi && zi)
                dxT[j] = d[0][k] + ty * (c[k] - cy[k]) - tz * (b[k + 1] - b[k]);
            if (xi && zi)
                dyT[j] = d[1][k] + tz * (a[k + 1] - a[k]) - tx * (c[k] - cx[k]);
            if (xi && yi)
                dzT[j] = d[2][k] + tx * (b[k + 1] - bx[k]) - ty * (a[k + 1] - ay[k]);
        }
}

struct ETriplet {
    float *t[3];
    const float *e0[3], *e1[3], *d0[3], *d1[3], *d2[3];
};

__global__ void __launch_bounds__(TILE_THREADS) compat_e_kernel(ETriplet a, const float *sigma,
                                                         const float *eps_i,
                                                         const float *eps_s,
                                                         const float *tau_d)
{
    pdl_begin();
    const int nx = c_sym.nx, ny = c_sym.ny, nz = c_sym.nz;
    const TileXY t(nx, blockDim.x, blockDim.y);
    const int x = t.x0 + threadIdx.x, y = t.y0 + threadIdx.y, z = blockIdx.y;
    if (x >= nx || y >= ny)
        return;
    // ex: x 0..nx-2, y 1..ny-2, z 1..nz-2; ey, ez: x 1..nx-1, y 0..ny-1, z 1..nz-1 (:147-175)
    const bool ex_on = x < nx - 1 && y >= 1 && y < ny - 1 && z >= 1 && z < nz - 1;
    const bool eyz_on = x >= 1 && z >= 1;
    if (!ex_on && !eyz_on)
        return;
    const size_t i = cell_index(x, y, z, nx, ny);
    // all 19 loads before the first store: with each component loaded, updated
    // and stored in turn the kernel ran 184 us on 256 x 256 x 200 (6.3 TB/s on its
    // 88 bytes per cell), so 162 (7.1 TB/s); two or four planes per thread gave
    // nothing more
    const float s = sigma[i], es = eps_s[i], ei = eps_i[i], tau = tau_d[i];
    float v[3][5];
#pragma unroll
    for (int c = 0; c < 3; c++)
        if (c == 0 ? ex_on : eyz_on) {
            v[c][0] = a.e0[c][i];
            v[c][1] = a.e1[c][i];
            v[c][2] = a.d0[c][i];
            v[c][3] = a.d1[c][i];
            v[c][4] = a.d2[c][i];
        }
    const DebyeCoef k = cell_coef(c_sym.dt, c_sym.eps0, s, es, ei, tau, FDTD_SCHEME_REFERENCE);
#pragma unroll
    for (int c = 0; c < 3; c++)
        if (c == 0 ? ex_on : eyz_on)
            a.t[c][i] = debye_update(k, v[c][0], v[c][1], v[c][2], v[c][3], v[c][4]);
}

__global__ void compat_sources_kernel(float *dzT, const float *dzS,
                                      const float *hx, const float *hy, int iter)
{
    pdl_begin();
    const int s = threadIdx.x;
    if (s >= c_sym.nsources)
        return;
    const int nx = c_sym.nx, ny = c_sym.ny;
    const int x = c_sym.sources[3 * s], y = c_sym.sources[3 * s + 1], z = c_sym.sources[3 * s + 2];
    const size_t i = cell_index(x, y, z, nx, ny);
    const float jz = (iter >= 0 && iter < c_sym.njz) ? g_jz[iter] : 0.0f;
    dzT[i] = dzS[i] + c_sym.dt / c_sym.dx * (hy[i] - hy[i - 1]) - c_sym.dt / c_sym.dy * (hx[i] - hx[i - nx]) - jz;
}

struct MurArgs {
    float *t[3];
    const float *s[3];
    MurSlabs rp;
};

// Face set blockIdx.z; x runs along its faster in-face axis, each thread takes
// MUR_ROWS rows of the other, gridDim.y apart, loads before stores.
constexpr int MUR_THREADS = 128, MUR_ROWS = 4;

__global__ void __launch_bounds__(MUR_THREADS) compat_mur_kernel(MurArgs a)
{
    pdl_begin();
    const int nx = c_sym.nx, ny = c_sym.ny, nz = c_sym.nz;
    const int f = blockIdx.z;
    const MurFace m = mur_face(f, nx, ny, nz);
    const int iu = blockIdx.x * MUR_THREADS + threadIdx.x;
    for (int iv = blockIdx.y; iv < m.len_v; iv += MUR_ROWS * gridDim.y)
        mur_apply_k<MUR_ROWS>(f, iu, iv, gridDim.y, m.len_v, nx, ny, nz, nx, c_sym.dt, c_sym.dx, c_sym.dy, c_sym.dz,
                              c_sym.mu0 * c_sym.eps0, a.rp, a.t[0], a.t[1], a.t[2], a.s[0], a.s[1], a.s[2], false);
}

int prologue(SymbolBlock *sym)
{
    int dev;
    int st = current_device_checked(&dev);
    if (st != FDTD_OK)
        return st;
    if (!g_symbols_ready[dev].load())
        return FDTD_ERR_NO_SYMBOLS;
    *sym = g_host_sym[dev];
    return FDTD_OK;
}

// The cells in columns of `planes` z planes.
dim3 cell_grid(const SymbolBlock &s, int planes)
{
    const dim3 t = cell_tile(s.nx);
    return tile_grid(s.nx, s.ny, s.nz, t.x, t.y, planes);
}

}  // namespace
}  // namespace fdtd

using namespace fdtd;

extern "C" {

int fdtd_copy_symbols(const FdtdParams *p)
{
    if (!p || p->nx < 3 || p->ny < 3 || p->nz < 3 || p->sourcesCount < 0 || p->sourcesCount > FDTD_MAX_SOURCES ||
        (p->sourcesCount > 0 && !p->sources) || p->jzCount < 0 || (p->jzCount > 0 && !p->jz))
        return FDTD_ERR_INVALID;
    if ((long long)p->nx * p->ny * p->nz > (1LL << 40) || p->nz > 65535)
        return FDTD_ERR_INVALID;
    for (int s = 0; s < p->sourcesCount; s++) {
        const int *q = p->sources + 3 * s;
        // updateSources reads hy at x-1 and hx at y-1 (:206-207).
        if (q[0] < 1 || q[0] >= p->nx || q[1] < 1 || q[1] >= p->ny || q[2] < 0 || q[2] >= p->nz)
            return FDTD_ERR_INVALID;
    }
    int dev;
    int st = current_device_checked(&dev);
    if (st != FDTD_OK)
        return st;
    SymbolBlock s{};
    s.nx = p->nx; s.ny = p->ny; s.nz = p->nz;
    s.dt = p->dt; s.dx = p->dx; s.dy = p->dy; s.dz = p->dz;
    s.mu0 = p->mu0; s.eps0 = p->eps0;
    s.nsources = p->sourcesCount;
    for (int k = 0; k < 3 * p->sourcesCount; k++)
        s.sources[k] = p->sources[k];
    s.njz = p->jzCount < FDTD_JZ_LEN ? p->jzCount : FDTD_JZ_LEN;
    cudaError_t e = cudaMemcpyToSymbol(c_sym, &s, sizeof s);
    if (e == cudaSuccess && s.njz > 0)
        e = cudaMemcpyToSymbol(g_jz, p->jz, sizeof(float) * s.njz);
    if (e != cudaSuccess)
        return e;
    g_host_sym[dev] = s;
    g_symbols_ready[dev].store(true);
    return FDTD_OK;
}

int fdtd_update_h(float *hx, float *hy, float *hz, const float *exSource, const float *eySource,
                  const float *ezSource, fdtd_stream_t stream)
{
    SymbolBlock s;
    int st = prologue(&s);
    if (st != FDTD_OK)
        return st;
    if (!hx || !hy || !hz || !exSource || !eySource || !ezSource)
        return FDTD_ERR_INVALID;
    return launch_pdl(false, compat_h_kernel, cell_grid(s, H_PLANES), cell_tile(s.nx), stream, hx, hy, hz, exSource, eySource,
                      ezSource);
}

int fdtd_update_d(float *dxTarget, float *dyTarget, float *dzTarget, const float *dxSource, const float *dySource,
                  const float *dzSource, const float *hx, const float *hy, const float *hz, fdtd_stream_t stream)
{
    SymbolBlock s;
    int st = prologue(&s);
    if (st != FDTD_OK)
        return st;
    if (!dxTarget || !dyTarget || !dzTarget || !dxSource || !dySource || !dzSource || !hx || !hy || !hz)
        return FDTD_ERR_INVALID;
    return launch_pdl(false, compat_d_kernel, cell_grid(s, D_PLANES), cell_tile(s.nx), stream, dxTarget, dyTarget, dzTarget,
                      dxSource, dySource, dzSource, hx, hy, hz);
}

int fdtd_update_e(float *exTarget, float *eyTarget, float *ezTarget, const float *exSource0, const float *eySource0,
                  const float *ezSource0, const float *exSource1, const float *eySource1, const float *ezSource1,
                  const float *dxSource0, const float *dySource0, const float *dzSource0, const float *dxSource1,
                  const float *dySource1, const float *dzSource1, const float *dxSource2, const float *dySource2,
                  const float *dzSource2, const float *sigma, const float *epsI, const float *epsS, const float *tauD,
                  fdtd_stream_t stream)
{
    SymbolBlock s;
    int st = prologue(&s);
    if (st != FDTD_OK)
        return st;
    ETriplet a{{exTarget, eyTarget, ezTarget},
               {exSource0, eySource0, ezSource0},
               {exSource1, eySource1, ezSource1},
               {dxSource0, dySource0, dzSource0},
               {dxSource1, dySource1, dzSource1},
               {dxSource2, dySource2, dzSource2}};
    for (int c = 0; c < 3; c++)
        if (!a.t[c] || !a.e0[c] || !a.e1[c] || !a.d0[c] || !a.d1[c] || !a.d2[c])
            return FDTD_ERR_INVALID;
    if (!sigma || !epsI || !epsS || !tauD)
        return FDTD_ERR_INVALID;
    return launch_pdl(false, compat_e_kernel, cell_grid(s, 1), cell_tile(s.nx), stream, a, sigma, epsI, epsS, tauD);
}

int fdtd_update_sources(float *dzTarget, const float *dzSource, const float *hx, const float *hy, int currIteration,
                        fdtd_stream_t stream)
{
    SymbolBlock s;
    int st = prologue(&s);
    if (st != FDTD_OK)
        return st;
    if (!dzTarget || !dzSource || !hx || !hy)
        return FDTD_ERR_INVALID;
    if (s.nsources == 0)
        return FDTD_OK;
    return launch_pdl(false, compat_sources_kernel, dim3(1), dim3(32), stream, dzTarget, dzSource, hx, hy, currIteration);
}

int fdtd_update_mur(float *exTarget, float *eyTarget, float *ezTarget, const float *exSource, const float *eySource,
                    const float *ezSource, const float *rpx0, const float *rpy0, const float *rpz0,
                    const float *rpxEnd, const float *rpyEnd, const float *rpzEnd, fdtd_stream_t stream)
{
    SymbolBlock s;
    int st = prologue(&s);
    if (st != FDTD_OK)
        return st;
    MurArgs a{{exTarget, eyTarget, ezTarget}, {exSource, eySource, ezSource}, {rpx0, rpy0, rpz0, rpxEnd, rpyEnd, rpzEnd}};
    for (int c = 0; c < 3; c++)
        if (!a.t[c] || !a.s[c])
            return FDTD_ERR_INVALID;
    if (!rpx0 || !rpy0 || !rpz0 || !rpxEnd || !rpyEnd || !rpzEnd)
        return FDTD_ERR_INVALID;
    int most_u = 1, most_v = 1;
    for (int f = 0; f < 12; f++) {
        const MurFace m = mur_face(f, s.nx, s.ny, s.nz);
        most_u = std::max(most_u, m.len_u);
        most_v = std::max(most_v, m.len_v);
    }
    const int rows = (most_v + MUR_ROWS - 1) / MUR_ROWS;
    const dim3 grid((unsigned)((most_u + MUR_THREADS - 1) / MUR_THREADS), (unsigned)std::min(rows, 65535), 12);
    return launch_pdl(false, compat_mur_kernel, grid, dim3(MUR_THREADS), stream, a);
}

}  // extern "C"
