// Matrix products of two run-time tensors on the CUDA cores: tosa.matmul on bf16 / f32 (products and sums rounded in index
// order of k, which the tensor cores do not do) and on int8 / int16 (int32 accumulation with wrap-around,
// tests/testdata/tosa_ops/matmul-in-int8-out-int32.mlir, matmul-in-int16-out-int16.mlir).
//
// A block computes a tile of the result in stages of KC values of k: both operands are staged [row][k] in shared memory, two stages,
// and while TX x TY threads multiply one of them the block's other threads (LOADERS) fill the next; the first stage is
// everybody's. The second operand may come as [N, K] (TB: a transpose in front of the product that the planner folded in).
// What bounds it: reading operands back. A 16-byte read returns 512 bytes to a warp, four cycles of the SM's path whether lanes share
// the value or not, so RM x RN results per thread, not the warp's shape, set the rate; bf16 is staged as it is and halves it. The
// row pitch of 16 bytes more puts the rows eight lanes read into different banks; a step's operands are read during the step before. Cold
// instructions are the other part: a launch runs each line of its code a few times, so loops stay rolled (an unrolled form
// with a register prefetch spent 3000 of 14000 cycles on fetching a stage that takes 1500 here).
// bf16, kernel alone: 512 x 64 x 512 4.1 -> 3.5 us, 512 x 512 x 64 8.6 -> 5.7 us (the order of k makes it a chain of 512 multiply-adds); f32
// 765 x 136 x 765 15.2 -> 13.3, 765 x 765 x 136 24.2 -> 23.0; one attention head of 512 x 64, three launches: 17.1 -> 12.3.
#include <cuda_bf16.h>

#include <atomic>

#include "../../include/torq_b200_ops.h"
#include "dependent_launch.cuh"
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
__device__ __forceinline__ void load4(const T* p, T (&v)[4]) {
  if (sizeof(T) == 2) {
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
    v[0] = (T)(q.x & 0xffff); v[1] = (T)(q.x >> 16); v[2] = (T)(q.y & 0xffff); v[3] = (T)(q.y >> 16);
  } else {
    const uint32_t q = __ldg(reinterpret_cast<const uint32_t*>(p));
    v[0] = (T)(q & 0xff); v[1] = (T)((q >> 8) & 0xff); v[2] = (T)((q >> 16) & 0xff); v[3] = (T)(q >> 24);
  }
}

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
// What a stage holds: bf16 as it is (reading operands back is what bounds the small products), everything else as its accumulator's type.
template <typename T> struct StagedOf { typedef typename AccOf<T>::type type; };
template <> struct StagedOf<uint16_t> { typedef uint16_t type; };

// value i of sixteen staged bytes; HALF: bf16
template <typename Acc, bool HALF>
__device__ __forceinline__ Acc value_of(const uint4& q, int i) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  if constexpr (HALF) return __uint_as_float(i & 1 ? w[i >> 1] & 0xffff0000u : w[i >> 1] << 16);
  else if constexpr (sizeof(Acc) == sizeof(float) && (Acc)0.5f != (Acc)0) return __uint_as_float(w[i]);
  else return (Acc)w[i];
}

// An operand's part of a stage, on its way from memory to shared memory as [row][k]: kRows x KC values in units of 16 bytes of a row of
// the operand, one load where they are aligned (vec). Zeros outside the operand (for integers too, which carry a zero point: what
// lies outside must add nothing). COLS: the operand is stored [K, rows]. kFlight units a thread are in registers between load and store.
template <typename TIn, bool COLS, int kRows, int KC>
struct StageCopy {
  typedef typename StagedOf<TIn>::type Staged;
  static constexpr int U = 16 / (int)sizeof(TIn), V = 16 / (int)sizeof(Staged), kPitch = KC + V, kFlight = 4, kUnits = kRows * KC / U;
  union { uint4 v; TIn e[U]; } r[kFlight];
  static __device__ __forceinline__ int row_of(int q) { return COLS ? q / KC * U : q / (KC / U); }
  static __device__ __forceinline__ int k_of(int q) { return COLS ? q % KC : q % (KC / U) * U; }
  // kn: values of k that are read, a multiple of 16
  __device__ __forceinline__ void load(const TIn* __restrict__ p, int row0, int rows, int k0, int K, int kn, bool vec, int q0, int n) {
#pragma unroll
    for (int i = 0; i < kFlight; i++) {
      const int q = q0 + i * n, row = row_of(q), k = k_of(q);
      r[i].v = make_uint4(0, 0, 0, 0);
      if (q >= kUnits || k >= kn) continue;
      const TIn* s = COLS ? p + (size_t)(k0 + k) * rows + row0 + row : p + (size_t)(row0 + row) * K + k0 + k;
      if (vec) {
        if (row0 + row < rows && k0 + k < K) r[i].v = __ldg(reinterpret_cast<const uint4*>(s));
      } else {
#pragma unroll
        for (int e = 0; e < U; e++)
          if (row0 + row + (COLS ? e : 0) < rows && k0 + k + (COLS ? 0 : e) < K) r[i].e[e] = __ldg(s + e);
      }
    }
  }
  __device__ __forceinline__ void store(Staged* to, int k0, int K, int kn, int zp, int q0, int n) {
#pragma unroll
    for (int i = 0; i < kFlight; i++) {
      const int q = q0 + i * n, row = row_of(q), k = k_of(q);
      if (q >= kUnits || k >= kn) continue;
      Staged w[U];
#pragma unroll
      for (int e = 0; e < U; e++) w[e] = k0 + k + (COLS ? 0 : e) < K ? (sizeof(Staged) == 2 ? (Staged)r[i].e[e] : (Staged)to_acc(r[i].e[e], zp)) : (Staged)0;
      if (COLS) {
#pragma unroll
        for (int e = 0; e < U; e++) to[(row + e) * kPitch + k] = w[e];
      } else {
#pragma unroll
        for (int e = 0; e < U; e += V) *reinterpret_cast<uint4*>(to + row * kPitch + k + e) = *reinterpret_cast<const uint4*>(w + e);
      }
    }
  }
};

template <typename TIn, typename TOut, bool TB, int RM, int RN, int TX, int TY, int KC, int LOADERS>
__global__ void __launch_bounds__(TX * TY + LOADERS) matmul_tile_kernel(const TIn* __restrict__ a, const TIn* __restrict__ b, TOut* __restrict__ out,
                                                                        int M, int K, int N, int n_tiles, int a_zp, int b_zp, int vec_a, int vec_b) {
  typedef typename AccOf<TIn>::type Acc;
  typedef typename StagedOf<TIn>::type Staged;
  constexpr int kPerLoad = 16 / (int)sizeof(Staged);
  constexpr int kTM = TY * RM, kTN = TX * RN, kPitch = KC + kPerLoad, kStage = (kTM + kTN) * kPitch;
  constexpr int kStep = RM * RN >= 16 && sizeof(Staged) == 4 ? 4 : 8;  // k of a step, whose operands are read during the step before
  extern __shared__ __align__(16) unsigned char tile_smem[];
  Staged* const smem = reinterpret_cast<Staged*>(tile_smem);  // two stages of kTM + kTN rows
  const int m0 = (int)(blockIdx.x / (unsigned)n_tiles) * kTM, n0 = (int)(blockIdx.x % (unsigned)n_tiles) * kTN;
  grid_dependency_wait();
  grid_dependency_release();
  auto load = [&](int k0, Staged* stage, int t, int n) {
    const int kn = min(KC, (K - k0 + 15) & ~15);
    StageCopy<TIn, false, kTM, KC> ca;
    StageCopy<TIn, !TB, kTN, KC> cb;
#pragma unroll 1
    for (int q0 = t; q0 < max(ca.kUnits, cb.kUnits); q0 += 4 * n) {
      ca.load(a, m0, M, k0, K, kn, vec_a != 0, q0, n);
      cb.load(b, n0, N, k0, K, kn, vec_b != 0, q0, n);
      ca.store(stage, k0, K, kn, a_zp, q0, n);
      cb.store(stage + kTM * kPitch, k0, K, kn, b_zp, q0, n);
    }
  };
  load(0, smem, threadIdx.x, TX * TY + LOADERS);
  __syncthreads();
  if (threadIdx.x >= TX * TY) {  // the loaders fill one buffer while the other one is multiplied
    for (int k0 = KC, s = 1; k0 < K; k0 += KC, s ^= 1) {
      load(k0, smem + s * kStage, (int)threadIdx.x - TX * TY, LOADERS);
      __syncthreads();
    }
    return;
  }
  // a warp computes 4 x 8 results (times RM x RN): its reads of a stage are then one wavefront each
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tx = warp % (TX / 8) * 8 + (lane & 7), ty = warp / (TX / 8) * 4 + (lane >> 3);
  Acc acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; i++)
#pragma unroll
    for (int j = 0; j < RN; j++) acc[i][j] = 0;
  for (int k0 = 0, s = 0; k0 < K; k0 += KC, s ^= 1) {
    const Staged* as = smem + s * kStage + ty * kPitch;
    const Staged* bs = smem + s * kStage + (kTM + tx) * kPitch;
    struct Operands {
      uint4 a[RM][kStep / kPerLoad], b[RN][kStep / kPerLoad];
    } even, odd;
    auto read = [&](Operands& o, int k) {
#pragma unroll
      for (int e = 0; e < kStep / kPerLoad; e++) {
#pragma unroll
        for (int i = 0; i < RM; i++) o.a[i][e] = *reinterpret_cast<const uint4*>(as + i * TY * kPitch + k + e * kPerLoad);
#pragma unroll
        for (int j = 0; j < RN; j++) o.b[j][e] = *reinterpret_cast<const uint4*>(bs + j * TX * kPitch + k + e * kPerLoad);
      }
    };
    auto multiply = [&](const Operands& o) {
#pragma unroll
      for (int e = 0; e < kStep; e++)
#pragma unroll
        for (int i = 0; i < RM; i++)
#pragma unroll
          for (int j = 0; j < RN; j++) acc[i][j] = mac(acc[i][j], value_of<Acc, sizeof(Staged) == 2>(o.a[i][e / kPerLoad], e % kPerLoad), value_of<Acc, sizeof(Staged) == 2>(o.b[j][e / kPerLoad], e % kPerLoad), TIn{});
    };
    const int kn = min(KC, (K - k0 + kStep - 1) & ~(kStep - 1));
    read(even, 0);
#pragma unroll 1
    for (int k = 0; k < kn; k += 2 * kStep) {
      if (k + kStep < kn) read(odd, k + kStep);
      multiply(even);
      if (k + kStep >= kn) break;
      if (k + 2 * kStep < kn) read(even, k + 2 * kStep);
      multiply(odd);
    }
    if (k0 + KC < K) __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RM; i++)
#pragma unroll
    for (int j = 0; j < RN; j++) {
      const int m = m0 + ty + TY * i, n = n0 + tx + TX * j;
      if (m < M && n < N) store_as(out + (size_t)m * N + n, acc[i][j]);
    }
}

// The same without loaders: 256 threads compute a (16 R) x (16 R) tile, 128 / R values of k at a time, every value staged as its accumulator's
// type; the next stage is fetched into registers while the current one is multiplied. Where there are blocks enough to fill the
// SMs, threads that only load cost more than they hide: run() says where.
template <typename TIn, typename TOut, bool TB, int R>
__global__ void __launch_bounds__(256) matmul_square_kernel(const TIn* __restrict__ a, const TIn* __restrict__ b, TOut* __restrict__ out,
                                                            int M, int K, int N, int n_tiles, int a_zp, int b_zp) {
  typedef typename AccOf<TIn>::type Acc;
  constexpr int T = 16 * R;
  constexpr int kKC = 128 / R;  // two groups of four elements per thread and operand whatever the tile
  constexpr int kPitch = kKC + 4;  // the eight rows a quarter-warp reads lie in different banks
  __shared__ __align__(16) Acc as[T][kPitch], bs[T][kPitch];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = (int)(blockIdx.x / (unsigned)n_tiles) * T, n0 = (int)(blockIdx.x % (unsigned)n_tiles) * T;
  constexpr int kPer = T * kKC / 4 / 256;  // groups of four elements per thread, operand and stage
  const bool ka = (K & 3) == 0, na = (N & 3) == 0;  // four elements of a row are aligned to their size (the operands are: run())
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

// whether an operand's rows can be read 16 bytes at a time
template <typename TIn, bool TB>
void aligned_rows(const void* a, const void* b, int K, int N, int& rows_a, int& rows_b) {
  rows_a = ((K * (int)sizeof(TIn)) & 15) == 0 && ((uintptr_t)a & 15) == 0;
  rows_b = (((TB ? K : N) * (int)sizeof(TIn)) & 15) == 0 && ((uintptr_t)b & 15) == 0;
}

template <typename TIn, typename TOut, bool TB, int R>
cudaError_t launch_square(const void* a, const void* b, void* out, int M, int K, int N, int a_zp, int b_zp, cudaStream_t stream) {
  constexpr int T = 16 * R;
  const long long tiles = (long long)((M + T - 1) / T) * ((N + T - 1) / T);
  return launch_dependent_if(false, matmul_square_kernel<TIn, TOut, TB, R>, dim3((unsigned)tiles), dim3(256), 0, stream, (const TIn*)a, (const TIn*)b, (TOut*)out, M, K, N,
                             (N + T - 1) / T, a_zp, b_zp);
}

template <typename TIn, typename TOut, bool TB, int RM, int RN, int TX, int TY, int KC, int LOADERS>
cudaError_t launch_tiles(const void* a, const void* b, void* out, int M, int K, int N, int a_zp, int b_zp, cudaStream_t stream) {
  auto kernel = matmul_tile_kernel<TIn, TOut, TB, RM, RN, TX, TY, KC, LOADERS>;
  constexpr int kTM = TY * RM, kTN = TX * RN, kSmem = 2 * (kTM + kTN) * (KC * (int)sizeof(typename StagedOf<TIn>::type) + 16), kOnePerSm = kSmem > 116 * 1024 ? kSmem : 116 * 1024;
  static std::atomic<unsigned long long> attr_done{0};
  if (first_use_on_device(attr_done)) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kOnePerSm);
    if (e != cudaSuccess) return e;
    mark_used_on_device(attr_done);
  }
  const long long tiles = (long long)((M + kTM - 1) / kTM) * ((N + kTN - 1) / kTN);
  int vec_a, vec_b;
  aligned_rows<TIn, TB>(a, b, K, N, vec_a, vec_b);
  // one grid dimension: the second ends at 65535 tiles
  // Launched early where every block has an SM to itself, and then made to take one: blocks that arrive while the kernel ahead still
  // runs are put wherever there is room, two or three to an SM beside empty ones (765 x 765 x 136: 23 -> 31 us).
  const bool early = tiles <= current_sm_count();
  return launch_dependent_if(early, kernel, dim3((unsigned)tiles), dim3(TX * TY + LOADERS), early ? kOnePerSm : kSmem, stream, (const TIn*)a, (const TIn*)b, (TOut*)out, M, K, N,
                          (N + kTN - 1) / kTN, a_zp, b_zp, vec_a, vec_b);
}

// With loaders: the largest tile of which there are two for every SM (64 x 32) or one for every other SM (32 x 32); 16 x 16 for what is
// smaller. More loaders where the stage holds two-byte values: rows that are not aligned are read value by value (measured with 128 / 256 / 384: 512 x 512 x 64 bf16
// 7.4 / 8.1 / 6.9 us, 511 x 511 x 61 12.2 / 10.6 / 8.8; 1023 x 1023 x 253 in 32 x 32 49 / 36; f32 there 44 / 60).
template <typename TIn, typename TOut>
cudaError_t run(const void* a, const void* b, void* out, int M, int K, int N, int a_zp, int b_zp, bool tb, cudaStream_t stream) {
  auto tiles = [&](int tm, int tn) { return (long long)((M + tm - 1) / tm) * ((N + tn - 1) / tn); };
  const int sms = current_sm_count();
  constexpr bool kHalf = sizeof(typename StagedOf<TIn>::type) == 2;
#define TB200_TILES(RM, RN, TX, TY, KC, LOADERS)                                                                        \
  return tb ? launch_tiles<TIn, TOut, true, RM, RN, TX, TY, KC, LOADERS>(a, b, out, M, K, N, a_zp, b_zp, stream)        \
            : launch_tiles<TIn, TOut, false, RM, RN, TX, TY, KC, LOADERS>(a, b, out, M, K, N, a_zp, b_zp, stream)
#define TB200_SQUARE(R)                                                                                   \
  return tb ? launch_square<TIn, TOut, true, R>(a, b, out, M, K, N, a_zp, b_zp, stream)                   \
            : launch_square<TIn, TOut, false, R>(a, b, out, M, K, N, a_zp, b_zp, stream)
  constexpr bool kFloat = sizeof(TIn) == 4;
  int vec_a, vec_b;
  if (tb) aligned_rows<TIn, true>(a, b, K, N, vec_a, vec_b);
  else aligned_rows<TIn, false>(a, b, K, N, vec_a, vec_b);
  const bool aligned = vec_a && vec_b, operands = (((uintptr_t)a | (uintptr_t)b) & 15) == 0;
  auto fills = [&](int stage) { return 3 * ((long long)(K + stage - 1) / stage * stage) <= 4ll * K; };  // its stages: multiplied to their end
  // Where the kernel without loaders is taken (us per launch, one behind the other, with loaders -> without):
  //   f32 in 64 x 64, from one tile an SM on. A multiplication and an addition per product leave no issue slots that loaders could fill:
  //   2048 x 1024 x 2048 458 -> 377, transposed 434 -> 345; 1023 x 253 x 1023 37.5 -> 31.4. Then 32 x 32 where rows are aligned: 640 x 640 x 640
  //   43.8 -> 38.0, transposed 45.2 -> 31.8 (1023 x 1023 x 253, which are not: 42.1 with, 45.9 without).
  //   The others in 64 x 64: rows that are not aligned (2047 x 1023 x 2047 i8 429 -> 397, transposed 401 -> 343; 1023 x 253 x 1023 bf16 30.8 -> 26.7);
  //   a short K (1024 x 32 x 1024 6.8 -> 5.7; bf16 transposed 1280 x 64 x 1280 11.9 -> 10.3, as it is 12.9 with and 15.5 without); and from four
  //   tiles an SM on a transposed operand (bf16 2048 x 1024 x 2048 313 -> 298) or a K of one stage, which leaves nothing to load ahead (8192 x 64 x
  //   2048 107 -> 99). Elsewhere loaders win: 2048 x 1024 x 2048 bf16 413 without, 329 with; 256 x 2048 x 8192 transposed 437 and 320.
  //   Integers in 32 x 32: transposed rows that are not aligned (1023 x 1023 x 253 i8 43.1 -> 37.0, i16 42.1 -> 35.4).
  // A K that leaves more than a quarter of its stages empty stays with loaders, which end at K: f32 transposed 765 x 136 x 765 13.3 with, 15.1 without.
  if (operands && fills(32) && tiles(64, 64) >= sms && (kFloat || !aligned || K <= (tb ? 64 : 32) || (tiles(64, 64) >= 4 * sms && (tb || K <= 64)))) TB200_SQUARE(4);
  if constexpr (!kHalf)
    if (operands && fills(64) && tiles(64, 64) < sms && tiles(32, 32) >= sms && (kFloat ? aligned : tb && !aligned)) TB200_SQUARE(2);
  if (tiles(64, 32) >= 2 * sms) TB200_TILES(4, 4, 8, 16, 64, 128);
  if (tiles(32, 32) >= sms / 2) TB200_TILES(2, 4, 8, 16, 64, (kHalf ? 256 : 128));
  TB200_TILES(1, 2, 8, 16, 256, (kHalf ? 384 : 256));
#undef TB200_TILES
#undef TB200_SQUARE
}

}  // namespace

cudaError_t launch_matmul_f(const void* a, const void* b, void* out, int M, int K, int N, int in_dtype, int out_dtype, bool b_transposed,
                     cudaStream_t stream) {
  if (in_dtype == TB200_BF16) {
    if (out_dtype == TB200_BF16) return run<uint16_t, uint16_t>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
    else return run<uint16_t, float>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
  } else {
    if (out_dtype == TB200_BF16) return run<float, uint16_t>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
    else return run<float, float>(a, b, out, M, K, N, 0, 0, b_transposed, stream);
  }
}

cudaError_t launch_matmul_int(const void* a, const void* b, void* out, bool in_i16, bool out_i16, int M, int K, int N, int a_zp,
                       int b_zp, bool b_transposed, cudaStream_t stream) {
  if (in_i16) {
    if (out_i16) return run<int16_t, int16_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
    else return run<int16_t, int32_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
  } else {
    if (out_i16) return run<int8_t, int16_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
    else return run<int8_t, int32_t>(a, b, out, M, K, N, a_zp, b_zp, b_transposed, stream);
  }
}

}  // namespace tb200
