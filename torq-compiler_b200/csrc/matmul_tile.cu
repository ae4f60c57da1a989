// Matrix products of two run-time tensors on the CUDA cores: tosa.matmul on bf16 / f32 (products and sums rounded in index
// order of k, which the tensor cores do not do) and on int8 / int16 (int32 accumulation with wrap-around,
// tests/testdata/tosa_ops/matmul-in-int8-out-int32.mlir, matmul-in-int16-out-int16.mlir).
//
// A block of 256 threads computes a (16 R) x (16 R) tile of the result. Both operands are staged [row][k] in shared memory,
// 128 / R values of k at a time, so that a thread takes four consecutive k of a row with one 16-byte read: 2 R reads for
// 4 R^2 multiply-adds. The row pitch of 4 words more puts the eight rows a quarter-warp reads into different banks. The next
// stage is fetched into registers while the current one is multiplied; a stage costs at least one L2 round trip, which is
// why the narrow tiles take long stages. The second operand may come as [N, K] (TB: a transpose in
// front of the product that the planner folded in).
// The sizes that occur (attention heads, a few hundred rows) are bound by latency, not by arithmetic: R is the largest
// tile that still gives every SM a block. bf16, [M, K] x [K, N]: 512 x 64 x 512 17.9 -> 4.1 us against one thread per output; 512 x 512 x 64
// 17.9 -> 8.8 us, one chain of 512 dependent multiply-adds per thread with two barriers per stage (issue slots 13 %, long and
// short scoreboard first).
#include <cuda_bf16.h>

#include "../../include/torq_b200_ops.h"
#include "kernels.h"

namespace tb200 {

namespace {

__device__ __forceinline__ float to_acc(float v, int) { return v; }
__device__ __forceinline__ float to_acc(uint16_t v, int) { return __uint_as_float((uint32_t)v << 16); }
__device__ __forceinline__ int to_acc(int8_t v, int zp) { return (int)v - zp; }
__device__ __forceinline__ int to_acc(int16_t v, int zp) { return (int)v - zp; }

// four consecutive elements (the pointer is aligned to them)
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 q = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <typename T>
__device__ __forceinline__ void load4_small(const T* p, T (&v)[4]) {
  if (sizeof(T) == 2) {
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
    v[0] = (T)(q.x & 0xffff); v[1] = (T)(q.x >> 16); v[2] = (T)(q.y & 0xffff); v[3] = (T)(q.y >> 16);
  } else {
    const uint32_t q = __ldg(reinterpret_cast<const uint32_t*>(p));
    v[0] = (T)(q & 0xff); v[1] = (T)((q >> 8) & 0xff); v[2] = (T)((q >> 16) & 0xff); v[3] = (T)(q >> 24);
  }
}
__device__ __forceinline__ void load4(const uint16_t* p, uint16_t (&v)[4]) { load4_small(p, v); }
__device__ __forceinline__ void load4(const int16_t* p, int16_t (&v)[4]) { load4_small(p, v); }
__device__ __forceinline__ void load4(const int8_t* p, int8_t (&v)[4]) { load4_small(p, v); }

// bf16 x bf16 products are exact in fp32, so one fused multiply-add rounds as a product and a sum do; f32 products round
__device__ __forceinline__ float mac(float acc, float a, float b, float) { return __fadd_rn(acc, __fmul_rn(a, b)); }
__device__ __forceinline__ float mac(float acc, float a, float b, uint16_t) { return fmaf(a, b, acc); }
template <typename T>
__device__ __forceinline__ int mac(int acc, int a, int b, T) { return (int)((uint32_t)acc + (uint32_t)a * (uint32_t)b); }

__device__ __forceinline__ void store_as(float* p, float v) { *p = v; }
__device__ __forceinline__ void store_as(uint16_t* p, float v) { *p = __bfloat16_as_ushort(__float2bfloat16_rn(v)); }
__device__ __forceinline__ void store_as(int32_t* p, int v) { *p = v; }
__device__ __forceinline__ void store_as(int16_t* p, int v) { *p = (int16_t)v; }

template <typename T> struct AccOf { typedef int type; };
template <> struct AccOf<float> { typedef float type; };
template <> struct AccOf<uint16_t> { typedef float type; };

template <typename TIn, typename TOut, bool TB, int R>
__global__ void __launch_bounds__(256) matmul_tile_kernel(const TIn* __restrict__ a, const TIn* __restrict__ b, TOut* __restrict__ out,
                                                          int M, int K, int N, int n_tiles, int a_zp, int b_zp) {
  typedef typename AccOf<TIn>::type Acc;
  constexpr int T = 16 * R;
  constexpr int kKC = 128 / R;  // k per stage: two groups of four elements per thread and operand whatever the tile
  constexpr int kPitch = kKC + 4;
  __shared__ __align__(16) Acc as[T][kPitch], bs[T][kPitch];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = (int)(blockIdx.x / (unsigned)n_tiles) * T, n0 = (int)(blockIdx.x % (unsigned)n_tiles) * T;
  constexpr int kQuads = T * kKC / 4;            // groups of four elements per operand and stage
  constexpr int kPer = kQuads / 256;             // per thread
  const bool ka = (K & 3) == 0, na = (N & 3) == 0;  // four elements of a row are aligned to their size
  TIn ra[kPer][4], rb[kPer][4];
  auto fetch_rows = [&](const TIn* p, int row0, int rows, int k0, TIn (&r)[kPer][4]) {  // operand stored [rows, K]
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      const int q = threadIdx.x + i * 256;
      const int row = row0 + q / (kKC / 4), k = k0 + (q % (kKC / 4)) * 4;
      const TIn* s = p + (size_t)row * K + k;
      if (row < rows && k + 3 < K && ka) {
        load4(s, r[i]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++) r[i][e] = row < rows && k + e < K ? s[e] : (TIn)0;
      }
    }
  };
  auto fetch_cols = [&](const TIn* p, int k0, TIn (&r)[kPer][4]) {  // operand stored [K, N]
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      const int q = threadIdx.x + i * 256;
      const int k = k0 + q % kKC, n = n0 + (q / kKC) * 4;
      const TIn* s = p + (size_t)k * N + n;
      if (k < K && n + 3 < N && na) {
        load4(s, r[i]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++) r[i][e] = k < K && n + e < N ? s[e] : (TIn)0;
      }
    }
  };
  auto fetch = [&](int k0) {
    fetch_rows(a, m0, M, k0, ra);
    if (TB) fetch_rows(b, n0, N, k0, rb);
    else fetch_cols(b, k0, rb);
  };
  // values beyond K must add nothing: integers carry a zero point, so what lies outside is stored as 0 after it
  auto put = [&](int k0) {
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      const int q = threadIdx.x + i * 256;
      {
        const int row = q / (kKC / 4), k = (q % (kKC / 4)) * 4;
#pragma unroll
        for (int e = 0; e < 4; e++) as[row][k + e] = k0 + k + e < K ? to_acc(ra[i][e], a_zp) : (Acc)0;
        if (TB) {
#pragma unroll
          for (int e = 0; e < 4; e++) bs[row][k + e] = k0 + k + e < K ? to_acc(rb[i][e], b_zp) : (Acc)0;
        }
      }
      if (!TB) {
        const int k = q % kKC, n = (q / kKC) * 4;
#pragma unroll
        for (int e = 0; e < 4; e++) bs[n + e][k] = k0 + k < K ? to_acc(rb[i][e], b_zp) : (Acc)0;
      }
    }
  };
  Acc acc[R][R];
#pragma unroll
  for (int i = 0; i < R; i++)
#pragma unroll
    for (int j = 0; j < R; j++) acc[i][j] = 0;
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += kKC) {
    __syncthreads();
    put(k0);
    __syncthreads();
    if (k0 + kKC < K) fetch(k0 + kKC);
#pragma unroll
    for (int k = 0; k < kKC; k += 4) {
      Acc av[R][4], bv[R][4];
#pragma unroll
      for (int i = 0; i < R; i++) {
        *reinterpret_cast<uint4*>(av[i]) = *reinterpret_cast<const uint4*>(&as[ty + 16 * i][k]);
        *reinterpret_cast<uint4*>(bv[i]) = *reinterpret_cast<const uint4*>(&bs[tx + 16 * i][k]);
      }
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int i = 0; i < R; i++)
#pragma unroll
          for (int j = 0; j < R; j++) acc[i][j] = mac(acc[i][j], av[i][e], bv[j][e], TIn{});
    }
  }
#pragma unroll
  for (int i = 0; i < R; i++)
#pragma unroll
    for (int j = 0; j < R; j++) {
      const int m = m0 + ty + 16 * i, n = n0 + tx + 16 * j;
      if (m < M && n < N) store_as(out + (size_t)m * N + n, acc[i][j]);
    }
}

template <typename TIn, typename TOut>
void run(const void* a, const void* b, void* out, int M, int K, int N, int a_zp, int b_zp, bool tb, cudaStream_t stream) {
  auto tiles = [&](int t) { return (long long)((M + t - 1) / t) * ((N + t - 1) / t); };
  const int sms = current_sm_count();
  auto go = [&](auto kern, int t) {
    // one grid dimension: the second ends at 65535 tiles
    kern<<<(unsigned)tiles(t), 256, 0, stream>>>((const TIn*)a, (const TIn*)b, (TOut*)out, M, K, N, (N + t - 1) / t, a_zp, b_zp);
  };
  if (tiles(64) >= sms) {
    if (tb) go(matmul_tile_kernel<TIn, TOut, true, 4>, 64);
    else go(matmul_tile_kernel<TIn, TOut, false, 4>, 64);
  } else if (tiles(32) >= sms) {
    if (tb) go(matmul_tile_kernel<TIn, TOut, true, 2>, 32);
    else go(matmul_tile_kernel<TIn, TOut, false, 2>, 32);
  } else {
    if (tb) go(matmul_tile_kernel<TIn, TOut, true, 1>, 16);
    else go(matmul_tile_kernel<TIn, TOut, false, 1>, 16);
  }
}

}  // namespace

void launch_matmul_f(const void* a, const void* b, void* out, int M, int K, int N, int in_dtype, int out_dtype, bool b_transposed,
                     cudaStream_t stream) {
  if (in_dtype == TB200_BF16) {
    if (out_dtype == TB200_BF16) run<uint16_t, uint16_t>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
    else run<uint16_t, float>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
  } else {
    if (out_dtype == TB200_BF16) run<float, uint16_t>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
    else run<float, float>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
  }
}

void launch_matmul_int(const void* a, const void* b, void* out, bool in_i16, bool out_i16, int M, int K, int N, int a_zp,
                       int b_zp, bool b_transposed, cudaStream_t stream) {
  if (in_i16) {
    if (out_i16) run<int16_t, int16_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
    else run<int16_t, int32_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
  } else {
    if (out_i16) run<int8_t, int16_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
    else run<int8_t, int32_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
  }
}

}  // namespace tb200
