// rows.cu -- dense host volumes to and from device arrays of padded rows.
//
// Solves keep their rows padded to a multiple of 16 cells so that TMA can
// address them; callers see dense volumes.  A strided copy
// (cudaMemcpy2DAsync) moves short rows slowly, the more so the shorter they
// are: 10 M floats to page-locked memory at 49 GB/s in rows of 61 and 115 in
// rows of 217, against 186 for one contiguous copy; bytes to the device at
// 15 - 58 GB/s against 590.  So the rows are packed by a kernel instead:
// straight into page-locked memory (183 GB/s, the link's rate, from 152
// blocks on), or through a device scratch area and contiguous copies (164
// GB/s into pageable memory).
#include <algorithm>

#include "rows.h"

namespace fdtd {
namespace {

constexpr int PACK_THREADS = 512;

// n elements of dense rows, from `first` on (an offset into the dense
// volume): consecutive threads write consecutive elements.
__global__ void __launch_bounds__(PACK_THREADS) pack_rows_kernel(float *__restrict__ dst,
                                                                 const float *__restrict__ src, size_t first, size_t n,
                                                                 unsigned nx, unsigned pitch)
{
    for (size_t i = blockIdx.x * (size_t)PACK_THREADS + threadIdx.x; i < n; i += (size_t)gridDim.x * PACK_THREADS) {
        const size_t row = (first + i) / nx;
        dst[i] = src[row * pitch + (first + i - row * nx)];
    }
}

__global__ void __launch_bounds__(PACK_THREADS) unpack_bytes_kernel(uint8_t *__restrict__ dst,
                                                                    const uint8_t *__restrict__ src, size_t n,
                                                                    unsigned nx, unsigned pitch)
{
    for (size_t i = blockIdx.x * (size_t)PACK_THREADS + threadIdx.x; i < n; i += (size_t)gridDim.x * PACK_THREADS) {
        const size_t row = i / nx;
        dst[row * pitch + (i - row * nx)] = src[i];
    }
}

unsigned blocks_for(size_t n, unsigned most)
{
    return (unsigned)std::min<size_t>((n + PACK_THREADS - 1) / PACK_THREADS, most);
}

// The device address of page-locked host memory [p, p + bytes), or null.
float *mapped_address(float *p, size_t bytes)
{
    cudaPointerAttributes a{}, z{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess ||
        cudaPointerGetAttributes(&z, reinterpret_cast<char *>(p) + bytes - 1) != cudaSuccess) {
        cudaGetLastError();  // not a sticky error: memory CUDA does not know
        return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || z.type != cudaMemoryTypeHost || !a.devicePointer || !z.devicePointer ||
        (size_t)(static_cast<char *>(z.devicePointer) - static_cast<char *>(a.devicePointer)) != bytes - 1)
        return nullptr;
    return static_cast<float *>(a.devicePointer);
}

}  // namespace

cudaError_t read_rows(float *host, const float *src, size_t rows, int nx, int pitch, float *scratch,
                      size_t scratch_floats, cudaStream_t s)
{
    const size_t n = rows * (size_t)nx;
    if (n == 0)
        return cudaSuccess;
    if (pitch == nx)
        return cudaMemcpyAsync(host, src, sizeof(float) * n, cudaMemcpyDeviceToHost, s);
    if (float *mapped = mapped_address(host, sizeof(float) * n)) {
        pack_rows_kernel<<<blocks_for(n, 152), PACK_THREADS, 0, s>>>(mapped, src, 0, n, nx, pitch);
        return cudaGetLastError();
    }
    if (!scratch || scratch_floats == 0)
        return cudaMemcpy2DAsync(host, sizeof(float) * nx, src, sizeof(float) * pitch, sizeof(float) * nx, rows,
                                 cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaSuccess;
    for (size_t o = 0; o < n && e == cudaSuccess; o += scratch_floats) {
        const size_t m = std::min(scratch_floats, n - o);
        pack_rows_kernel<<<blocks_for(m, 152 * 4), PACK_THREADS, 0, s>>>(scratch, src, o, m, nx, pitch);
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(host + o, scratch, sizeof(float) * m, cudaMemcpyDeviceToHost, s);
    }
    return e;
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
    unpack_bytes_kernel<<<blocks_for(n, 152 * 4), PACK_THREADS, 0, s>>>(dst, scratch, n, nx, pitch);
    return cudaGetLastError();
}

}  // namespace fdtd
