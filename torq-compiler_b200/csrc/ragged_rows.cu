// Rows whose length is no multiple of 16 bytes (odd channel counts, odd K). The copy engine and 16-byte loads need rows at a
// 16-byte pitch, and without them such a layer ran on the CUDA cores. Copying the rows to a padded pitch first, and cutting
// a padded result back afterwards, costs two passes over small tensors and a launch each, and the product itself runs on the
// tensor cores. FullyConnected 3000 x 4001 -> 4003: 3766 -> 57 us; 3x3, 64 x
// 28 x 28 x 100 -> 100 at stride 2: 51 -> 22 us.
// Bound by memory: a thread makes 16 bytes from five aligned words (neighbours share them in L1). Only words that hold bytes
// of the tensor are touched.
#include "dependent_launch.cuh"
#include "device_memory.cuh"
#include "kernels.h"

namespace tb200 {
namespace {

// out[r][0 .. pitch) <- x[r][0 .. K) followed by unspecified bytes (they meet zero weights); pitch a multiple of 16
__global__ void __launch_bounds__(256) pad_rows_kernel(const int8_t* x, int8_t* out, long long rows, int K, int pieces) {
  grid_dependency_wait();
  grid_dependency_release();
  const long long n = rows * pieces, total = rows * K, stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    long long r;
    int c;
    if (n < (1ll << 32)) { r = (uint32_t)i / (uint32_t)pieces; c = (int)((uint32_t)i - (uint32_t)r * (uint32_t)pieces); }
    else { r = i / pieces; c = (int)(i - r * pieces); }
    reinterpret_cast<uint4*>(out)[i] = load16_any(x, r * K + 16 * c, total);
  }
}

// out[r][0 .. N) <- x[r][0 .. N) with rows of x `pitch` (a multiple of 16) bytes apart; 16 bytes of the contiguous result per thread
__global__ void __launch_bounds__(256) trim_rows_kernel(const int8_t* x, int8_t* out, long long rows, int N, int pitch) {
  grid_dependency_wait();
  grid_dependency_release();
  const long long total = rows * N, n = (total + 15) >> 4, src_total = rows * pitch, stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const long long f = i << 4;
    long long r;
    int c;
    if (total < (1ll << 32)) { r = (uint32_t)f / (uint32_t)N; c = (int)((uint32_t)f - (uint32_t)r * (uint32_t)N); }
    else { r = f / N; c = (int)(f - r * N); }
    uint4 v;
    if (c + 16 <= N) {
      v = load16_any(x, r * pitch + c, src_total);
    } else {
      uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 16; j++) {
        if (f + j < total) w[j >> 2] |= (uint32_t)(uint8_t)x[r * pitch + c] << (8 * (j & 3));
        if (++c == N) { c = 0; r++; }
      }
      v = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (f + 16 <= total) {
      reinterpret_cast<uint4*>(out)[i] = v;
    } else {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 16; j++)
        if (f + j < total) out[f + j] = (int8_t)(w[j >> 2] >> (8 * (j & 3)));
    }
  }
}

unsigned grid_of(long long threads) {
  const long long blocks = (threads + 255) / 256, most = 8ll * current_sm_count();
  return (unsigned)(blocks < 1 ? 1 : blocks < most ? blocks : most);
}

}  // namespace

void launch_pad_rows(const int8_t* x, int8_t* out, long long rows, int K, int pitch, cudaStream_t stream) {
  launch_dependent(pad_rows_kernel, dim3(grid_of(rows * (pitch / 16))), dim3(256), 0, stream, x, out, rows, K, pitch / 16);
}
void launch_trim_rows(const int8_t* x, int8_t* out, long long rows, int N, int pitch, cudaStream_t stream) {
  launch_dependent(trim_rows_kernel, dim3(grid_of((rows * N + 15) / 16)), dim3(256), 0, stream, x, out, rows, N, pitch);
}

}  // namespace tb200
