// rows.cu -- dense host volumes to and from device arrays of padded rows.
//
// Solves keep their rows padded to a multiple of 16 cells so that TMA can
// address them; callers see dense volumes.  A strided copy
// (cudaMemcpy2DAsync) moves short rows slowly, the more so the shorter they
// are: 10 M floats to page-locked memory at 49 GB/s in rows of 61 and 115 in
// rows of 217; bytes to the device at 15 - 58 GB/s against 590.  So the rows
// are packed by a kernel instead: straight into page-locked memory, or through
// a device scratch area and one contiguous copy.  The scratch area holds the
// whole volume: in pieces of 16 MB a read into fresh host pages took 33 ms on
// 301 x 245 x 187 and 18 - 235 on 497 x 500 x 300 (one piece 2.5 and 12.0, as
// copies of dense rows take), into pages in use 0.39 and 2.00 (0.34 and 1.68; dense
// 0.31 and 1.58).
//
// Page-locked memory is written by the kernel for long dense rows as well.  One
// contiguous copy of 420 MB ran at 107 - 191 GB/s, from one buffer and one
// moment to the next (now and then at a fifth of that); the kernel at 189 -
// 191 every time, the link's rate, with 16-byte stores from 76 blocks on
// (4-byte stores: 180 - 185).  Short ones go by the copy engine: reads of 0.13 /
// 1.0 / 4.2 / 16.8 / 52 / 420 MB took 21.7 / 28.0 / 44.5 / 110 / 294.8 / 2195 us
// so (in a quiet hour) and 25.5 / 30.3 / 46.8 / 112 / 296.7 / 2205 by the kernel.
#include <cuda.h>

#include <algorithm>

#include "rows.h"

namespace fdtd {
namespace {

constexpr int PACK_THREADS = 512;

unsigned blocks_for(size_t n, unsigned most)
{
    return (unsigned)std::min<size_t>((n + PACK_THREADS - 1) / PACK_THREADS, most);
}

// n elements of dense rows.  Each thread writes four at once, on 16 bytes: dst
// is `skew` elements above such a boundary, and the first and last group may be
// partial.
__global__ void __launch_bounds__(PACK_THREADS) pack_rows_kernel(float *__restrict__ dst,
                                                                 const float *__restrict__ src, size_t n, unsigned nx,
                                                                 unsigned pitch, unsigned skew)
{
    const size_t groups = (n + skew + 3) / 4;
    for (size_t g = blockIdx.x * (size_t)PACK_THREADS + threadIdx.x; g < groups; g += (size_t)gridDim.x * PACK_THREADS) {
        const size_t begin = g == 0 ? 0 : 4 * g - skew, end = min(4 * g + 4 - skew, n);
        const size_t row = begin / nx;
        unsigned x = (unsigned)(begin - row * nx);
        const float *p = src + row * pitch + x;
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (begin + k < end)
                v[k] = *p;
            if (++x == nx) {  // on to the next row
                x = 0;
                p += pitch - nx;
            }
            p++;
        }
        if (end - begin == 4) {
            *reinterpret_cast<float4 *>(dst + begin) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (begin + k < end)
                    dst[begin + k] = v[k];
        }
    }
}

void launch_pack(float *dst, const float *src, size_t n, int nx, int pitch, unsigned most, cudaStream_t s)
{
    const unsigned skew = (unsigned)(reinterpret_cast<uintptr_t>(dst) / sizeof(float) % 4);
    pack_rows_kernel<<<blocks_for((n + skew + 3) / 4, most), PACK_THREADS, 0, s>>>(dst, src, n, nx, pitch, skew);
}

// n elements of dense rows, out of padded rows or (UNPACK) into them.
template <class T, bool UNPACK>
__global__ void __launch_bounds__(PACK_THREADS) move_rows_kernel(T *__restrict__ dst, const T *__restrict__ src,
                                                                 size_t n, unsigned nx, unsigned pitch)
{
    for (size_t i = blockIdx.x * (size_t)PACK_THREADS + threadIdx.x; i < n; i += (size_t)gridDim.x * PACK_THREADS) {
        const size_t row = i / nx, j = row * pitch + (i - row * nx);
        if (UNPACK)
            dst[j] = src[i];
        else
            dst[i] = src[j];
    }
}

template <class T, bool UNPACK>
cudaError_t launch_move(T *dst, const T *src, size_t n, int nx, int pitch, cudaStream_t s)
{
    move_rows_kernel<T, UNPACK><<<blocks_for(n, 152 * 4), PACK_THREADS, 0, s>>>(dst, src, n, nx, pitch);
    return cudaGetLastError();
}

// A dense host volume to or from padded rows, through scratch.
template <class T>
cudaError_t move_block(void *dev, void *host, size_t n, int nx, int pitch, void *scratch, bool to_host, cudaStream_t s)
{
    T *rows = static_cast<T *>(dev), *dense = static_cast<T *>(scratch);
    if (to_host) {
        const cudaError_t e = launch_move<T, false>(dense, rows, n, nx, pitch, s);
        return e != cudaSuccess ? e : cudaMemcpyAsync(host, dense, sizeof(T) * n, cudaMemcpyDeviceToHost, s);
    }
    const cudaError_t e = cudaMemcpyAsync(dense, host, sizeof(T) * n, cudaMemcpyHostToDevice, s);
    return e != cudaSuccess ? e : launch_move<T, true>(rows, dense, n, nx, pitch, s);
}

// Whether a kernel may write host memory [p, p + bytes): floats on their own
// alignment, all within one page-locked allocation (the two ends alone do not
// tell: pages between two registered ranges need not be mapped) that the
// device sees at the same address.  Anything else is left to the copy engine.
bool kernel_may_write(const float *p, size_t bytes)
{
    using Get = CUresult (*)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
    static const Get get = []() -> Get {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<Get>(f);
    }();
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    unsigned type = 0, managed = 0;
    CUdeviceptr dev = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                  CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void *to[] = {&type, &managed, &dev, &start, &size};
    return get && at % sizeof(float) == 0 && get(5, what, to, (CUdeviceptr)at) == CUDA_SUCCESS &&
           type == CU_MEMORYTYPE_HOST && !managed && dev == (CUdeviceptr)at && start <= dev &&
           bytes <= size && dev - start <= size - bytes;
}

}  // namespace

cudaError_t pack_rows(float *dst, const float *src, size_t rows, int nx, int pitch, cudaStream_t s)
{
    launch_pack(dst, src, rows * (size_t)nx, nx, pitch, 152 * 4, s);
    return cudaGetLastError();
}

cudaError_t read_rows(float *host, const float *src, size_t rows, int nx, int pitch, float *scratch, cudaStream_t s)
{
    const size_t n = rows * (size_t)nx;
    if (n == 0)
        return cudaSuccess;
    if ((pitch != nx || sizeof(float) * n >= LONG_READ_BYTES) && kernel_may_write(host, sizeof(float) * n)) {
        launch_pack(host, src, n, nx, pitch, 152, s);
        return cudaGetLastError();
    }
    if (pitch == nx)
        return cudaMemcpyAsync(host, src, sizeof(float) * n, cudaMemcpyDeviceToHost, s);
    if (!scratch)
        return cudaMemcpy2DAsync(host, sizeof(float) * nx, src, sizeof(float) * pitch, sizeof(float) * nx, rows,
                                 cudaMemcpyDeviceToHost, s);
    const cudaError_t e = pack_rows(scratch, src, rows, nx, pitch, s);
    return e != cudaSuccess ? e : cudaMemcpyAsync(host, scratch, sizeof(float) * n, cudaMemcpyDeviceToHost, s);
}

cudaError_t write_byte_rows(uint8_t *dst, const uint8_t *host, size_t rows, int nx, int pitch, uint8_t *scratch,
                            cudaStream_t s)
{
    const size_t n = rows * (size_t)nx;
    if (pitch == nx)
        return cudaMemcpyAsync(dst, host, n, cudaMemcpyHostToDevice, s);
    const cudaError_t e = cudaMemcpyAsync(scratch, host, n, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess)
        return e;
    return launch_move<uint8_t, true>(dst, scratch, n, nx, pitch, s);
}

cudaError_t move_rows(void *dev, void *host, size_t elem, size_t rows, int nx, int pitch, void *scratch, bool to_host,
                      cudaStream_t s)
{
    const size_t n = rows * (size_t)nx;
    return elem == sizeof(uint16_t) ? move_block<uint16_t>(dev, host, n, nx, pitch, scratch, to_host, s)
                                    : move_block<uint32_t>(dev, host, n, nx, pitch, scratch, to_host, s);
}

}  // namespace fdtd
