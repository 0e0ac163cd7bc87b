// rows.h -- dense host volumes to and from device arrays of padded rows.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace fdtd {

// Row pitch of a grid's arrays: a multiple of 16 cells (TMA wants 16-byte
// strides of the class bytes too).  Rows below 16 cells stay as they are, so
// that padding never doubles a state.
inline int padded_rows_pitch(int nx) { return nx < 16 ? nx : (nx + 15) & ~15; }

// Row pitch of a single solve's arrays: padded where the padded rows' kernels
// gain by it and the memory is there.  us per step on dense and padded rows:
// * Compact forms: the strip kernel against the z-marching kernel fed by 4-byte
//   cp.async; 301 x 245 x 187 384 and 159, 17 x 300 x 300 100 and 53.
// * D form, the single-pass kernel (97 bytes per cell of a padded row) against
//   the two-pass kernels (121 per cell): 217 x 253 x 181 208 and 165, 49 x 300 x
//   300 (padding 1.31) 112 and 104, 36 (1.33) 100 and 101, 33 (1.45) 86 and 107, 17
//   (1.88) 50 and 59.  Up to 4/3.
// * Two-pass kernels need no TMA: 217 x 253 x 181 206 and 207, 44 x 300 x 300 103
//   and 109, 17 51 and 63.  Never.
// The padding, and the volume that stages reads of padded rows, may take a quarter
// of what dense rows would leave free (cell_bytes: the state's bytes per cell), so
// that monitors and other solves keep their room.
inline int solve_rows_pitch(int nx, size_t rows, bool two_pass, bool compact, size_t cell_bytes, size_t free_bytes)
{
    const int pitch = padded_rows_pitch(nx);
    if (two_pass || (!compact && 3ll * pitch > 4ll * nx))
        return nx;
    const size_t dense = rows * nx * cell_bytes, extra = rows * (pitch - nx) * cell_bytes + rows * nx * sizeof(float);
    return free_bytes > dense && extra <= (free_bytes - dense) / 4 ? pitch : nx;
}

// Dense rows from here on are read into page-locked memory by a kernel: it costs
// 0.6 % there (52 MB: 0.7 %), below up to 15 %.
constexpr size_t LONG_READ_BYTES = size_t(64) << 20;

// Queues on s the copy of `rows` rows of nx floats, pitch floats apart, into
// the dense host volume.  Page-locked memory is written by a kernel (short
// volumes of dense rows are copied), other memory through scratch (rows * nx
// floats of device memory that work on s may use; without it a strided copy;
// dense rows are copied as they are).
cudaError_t read_rows(float *host, const float *src, size_t rows, int nx, int pitch, float *scratch, cudaStream_t s);

// Queues on s the packing of such rows into device memory.
cudaError_t pack_rows(float *dst, const float *src, size_t rows, int nx, int pitch, cudaStream_t s);

// Queues on s the copy of a dense host byte volume into rows pitch bytes
// apart; scratch: rows * nx bytes of device memory (unused where pitch is nx).
cudaError_t write_byte_rows(uint8_t *dst, const uint8_t *host, size_t rows, int nx, int pitch, uint8_t *scratch,
                            cudaStream_t s);

// Queues on s the copy of a volume of 2- or 4-byte elements from padded rows
// on the device to a dense pageable host volume, or back (checkpoints), through
// scratch (rows * nx elements).  Strided copies of rows of 17 floats took five times as long as one
// copy of dense rows to the device, of 217 half as long again.
cudaError_t move_rows(void *dev, void *host, size_t elem, size_t rows, int nx, int pitch, void *scratch, bool to_host,
                      cudaStream_t s);

}  // namespace fdtd
