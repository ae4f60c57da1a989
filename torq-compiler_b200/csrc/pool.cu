// Pooling (torq_hl.maxpool2d, PoolingPattern.cpp:128-258; tosa.avg_pool2d).
//
// pool_strip_kernel takes the windows networks use (2x2 and 3x3 at stride 2, 3x3 and 5x5 at stride 1): a thread owns one
// output column of 4 or 16 channels (or one channel) and ROWS output rows, and keeps the horizontal reduction of the last
// K input rows in registers, so every input row is loaded and reduced once per strip. No divisions outside the prologue.
//  * Maximum on packed bytes: this machine has a full-rate max.s16x2 but no byte form (the byte intrinsics expand into
//    ~10 instructions), so a word is held as two halves whose bytes sit in the HIGH byte of 16-bit fields: (w << 8) for
//    bytes 0 and 2, w itself for bytes 1 and 3. The low byte of a field only breaks ties, never the high byte's maximum.
//  * Sum on packed bytes: bytes biased by 128 are summed as 16-bit fields (at most 25 * 255 each), two per addition.
//  * Average: the rescale depends only on the number of taps inside the image. The planner gives per count a record
//    {M', K} for which (sum * 2^16 * M' + K) >> 40 is TOSA's result for every sum that can occur (checked there); one
//    multiply-add, the result's byte is bits 8..15 of the high word, and the 16-bit saturating pack is the int8 clamp.
// 64x112x112x64, 3x3 stride 2 (64 MB; kernel alone): max with a table behind it 21 + a table pass -> 13.3 us, average 28 -> 15.8 us. What
// bounds it: the latency of its loads. A third of the warps fit (52 .. 64 registers), they wait for memory three quarters of
// the time, issue slots are 42 .. 50 % used and DRAM 28 .. 35 %.
//
// The kernels below it take every other window: one thread per output pixel and 16, 4 or 1 channels; avgpool_warp_kernel
// spreads the taps of a large window over a warp (the global pool at the end of a classifier).
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "dependent_launch.cuh"
#include "device_memory.cuh"
#include "kernels.h"

namespace tb200 {

namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(long long work_items, int per_block = kThreads) {
  long long blocks = (work_items + per_block - 1) / per_block;
  const long long cap = 148LL * 16;  // 148 SMs x resident blocks; the loops stride over the rest
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (unsigned)blocks;
}

constexpr int kStripThreads = 128;

// Sum and packed unsigned maximum of N words of two 16-bit fields (three operands to an instruction).
template <int N>
__device__ __forceinline__ uint32_t sum_of(const uint32_t (&v)[N]) {
  uint32_t s = v[0];
#pragma unroll
  for (int i = 1; i < N; i++) s += v[i];
  return s;
}
// The same for sums below 2048 on the other arithmetic pipe: the bit pattern of a 16-bit float below 2^-13 is its value in units of
// 2^-24, and sums of such floats are exact.
template <int N>
__device__ __forceinline__ uint32_t row_sum(const uint32_t (&v)[N]) {
  static_assert(N * 255 < 2048, "bit patterns count units only below 2048");
  uint32_t s = v[0];
#pragma unroll
  for (int i = 1; i < N; i++) asm("add.rn.f16x2 %0, %0, %1;" : "+r"(s) : "r"(v[i]));
  return s;
}
template <int N>
__device__ __forceinline__ uint32_t max_u16x2_of(const uint32_t (&v)[N]) {
  uint32_t m = v[0];
  int i = 1;
#pragma unroll
  for (; i + 1 < N; i += 2) m = __vimax3_u16x2(m, v[i], v[i + 1]);
  return i < N ? __vmaxu2(m, v[i]) : m;
}
template <int N>
__device__ __forceinline__ uint32_t max_s16x2_of(const uint32_t (&v)[N]) {
  uint32_t m = v[0];
  int i = 1;
#pragma unroll
  for (; i + 1 < N; i += 2) m = __vimax3_s16x2(m, v[i], v[i + 1]);
  return i < N ? max_s16x2(m, v[i]) : m;
}
__device__ __forceinline__ uint32_t pack_sat_s16x2(int lo, int hi) {
  uint32_t r;
  asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(r) : "r"(hi), "r"(lo));
  return r;
}

// VW: 32-bit words of channels per thread (4 or 1), or 0 for a single channel.
template <int VW, int K, int S, int ROWS, bool AVG, bool LUT>
__global__ void __launch_bounds__(kStripThreads) pool_strip_kernel(PoolArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ uint8_t lut_s[256];
  if (LUT) {
    for (int i = threadIdx.x; i < 256; i += kStripThreads) lut_s[i] = (uint8_t)a.lut[(int)(int8_t)i + 128];
    __syncthreads();
  }
  constexpr int VB = VW == 0 ? 1 : 4 * VW;  // channels per thread
  constexpr int NW = VW == 0 ? 1 : VW;
  const int groups = a.C / VB;
  const int col = blockIdx.x * kStripThreads + threadIdx.x;
  if (col >= a.OW * groups) return;
  const int ow = col / groups, g = col - ow * groups;
  const int oh0 = blockIdx.y * ROWS;
  const int iw0 = ow * S - a.pad_l, ih0 = oh0 * S - a.pad_t;
  const int8_t* img = a.x + (size_t)blockIdx.z * a.H * a.W * a.C + g * VB;
  int8_t* out = a.out + (((size_t)blockIdx.z * a.OH + oh0) * a.OW + ow) * a.C + g * VB;
  bool col_ok[K];
  int ncol = 0;
#pragma unroll
  for (int k = 0; k < K; k++) {
    col_ok[k] = iw0 + k >= 0 && iw0 + k < a.W;
    ncol += col_ok[k];
  }
  const uint32_t padw = (uint32_t)(a.pad_value & 0xff) * 0x01010101u;

  // horizontal reduction of one input row: e = bytes 0 and 2, o = bytes 1 and 3 of every word
  struct Row {
    uint32_t e[NW], o[NW];
  };
  auto load_row = [&](int ih) {
    Row r;
    const bool row_ok = ih >= 0 && ih < a.H;
    const int8_t* px = img + ((long long)ih * a.W + iw0) * a.C;
    uint32_t w[K][NW];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const bool ok = row_ok && col_ok[k];
#pragma unroll
      for (int j = 0; j < NW; j++) w[k][j] = AVG ? 0x80808080u : padw;  // outside: the pad value / nothing
      if (ok) {
        const int8_t* p = px + (size_t)k * a.C;
        if (VW == 4) {
          const uint4 v = *reinterpret_cast<const uint4*>(p);
          w[k][0] = v.x; w[k][NW > 1 ? 1 : 0] = v.y; w[k][NW > 2 ? 2 : 0] = v.z; w[k][NW > 3 ? 3 : 0] = v.w;
        } else if (VW == 1) {
          w[k][0] = *reinterpret_cast<const uint32_t*>(p);
        } else {
          w[k][0] = (uint32_t)(uint8_t)*p;
        }
      } else if (VW == 0) {
        w[k][0] = AVG ? 0x80u : padw & 0xffu;
      }
    }
#pragma unroll
    for (int j = 0; j < NW; j++) {
      if (AVG) {
        r.e[j] = r.o[j] = 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
          const uint32_t u = w[k][j] ^ 0x80808080u;
          r.e[j] += u & 0x00ff00ffu;
          if (VW != 0) r.o[j] += __byte_perm(u, 0, 0x4341);
        }
      } else {
        r.e[j] = w[0][j] << 8;
        r.o[j] = w[0][j];
#pragma unroll
        for (int k = 1; k < K; k++) {
          r.e[j] = max_s16x2(r.e[j], w[k][j] << 8);
          if (VW != 0) r.o[j] = max_s16x2(r.o[j], w[k][j]);
        }
      }
    }
    return r;
  };

  constexpr int NR = (ROWS - 1) * S + K;
  Row rows[NR];
#pragma unroll
  for (int i = 0; i < K - S; i++) rows[i] = load_row(ih0 + i);
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    if (oh0 + r >= a.OH) return;
#pragma unroll
    for (int i = 0; i < S; i++) rows[r * S + K - S + i] = load_row(ih0 + r * S + K - S + i);
    uint32_t res[NW];
    int count = 0;
    if (AVG) {
      const int top = ih0 + r * S;
      count = ncol * (min(top + K, a.H) - max(top, 0));
    }
    const int4 c = AVG ? __ldg(a.by_count + count) : make_int4(0, 0, 0, 0);
    const unsigned long long kk = ((unsigned long long)(uint32_t)c.w << 32) | (uint32_t)c.z;
#pragma unroll
    for (int j = 0; j < NW; j++) {
      uint32_t e = rows[r * S].e[j], o = rows[r * S].o[j];
#pragma unroll
      for (int i = 1; i < K; i++) {
        if (AVG) {
          e += rows[r * S + i].e[j];
          o += rows[r * S + i].o[j];
        } else {
          e = max_s16x2(e, rows[r * S + i].e[j]);
          o = max_s16x2(o, rows[r * S + i].o[j]);
        }
      }
      if (AVG) {
        const int h0 = (int)(((unsigned long long)(e << 16) * (uint32_t)c.x + kk) >> 32);
        const int h2 = (int)(((unsigned long long)(e & 0xffff0000u) * (uint32_t)c.x + kk) >> 32);
        const int h1 = (int)(((unsigned long long)(o << 16) * (uint32_t)c.x + kk) >> 32);
        const int h3 = (int)(((unsigned long long)(o & 0xffff0000u) * (uint32_t)c.x + kk) >> 32);
        res[j] = VW == 0 ? high_bytes4(h0, h0, h0, h0) : high_bytes4(h0, h1, h2, h3);
      } else {
        res[j] = VW == 0 ? (e >> 8) & 0xffu : __byte_perm(e, o, 0x7351);
      }
      if (LUT) res[j] = VW == 0 ? (uint32_t)lut_s[res[j] & 0xff] : lut_word(lut_s, res[j]);
    }
    if (VW == 4)
      *reinterpret_cast<uint4*>(out) = make_uint4(res[0], res[NW > 1 ? 1 : 0], res[NW > 2 ? 2 : 0], res[NW > 3 ? 3 : 0]);
    else if (VW == 1) *reinterpret_cast<uint32_t*>(out) = res[0];
    else *out = (int8_t)res[0];
    out += (size_t)a.OW * a.C;
  }
}

// add / sub of the max pool (with an optional table behind it) and the average pool of one tensor: one pass over the input where the
// three ops make three passes and move 2.25 times the bytes. A thread owns one output column of 16, 4 or 1 channels and a strip of
// rows; the rows the next step needs are loaded before the last ones are reduced. Both reductions work on the same unpacked bytes
// (biased by 128, two to a word as 16-bit fields: unsigned maxima and sums). What follows the maximum (table, factor and constant of
// the add's linear form) is one 64-bit entry per byte value, filled by the block before it waits for the launch ahead; the average's
// byte is multiplied in by one multiply-add.
// 64x112x112x64, 3x3 stride 2, table behind the maximum (kernel alone, buffers out of L2): three launches 39 us, this one 20.1. What bounds
// it: integer instructions, about 115 per four outputs and most of them on one pipe (measured: the sums of a row on the float pipe
// 20.7 -> 20.1; input staged in shared memory, which halves what L2 is asked for, 27; all loads of a strip up front and no loop 22.5).
// Four rows to a strip: 1, 2, 3, 4, 7, 14 rows take 29, 22.9, 21.0, 20.1, 20.5, 23.6 us (halo rows against waves of blocks).
template <int VW, int K, int S>
__global__ void __launch_bounds__(kStripThreads, VW == 4 ? 4 : 7) pool_add_kernel(const PoolAddArgs pa, int cols, int strips, int strip_rows, int threads) {
  const PoolArgs& a = pa.pool;
  __shared__ long long from_max[256];
  for (int v = threadIdx.x; v < 256; v += kStripThreads) {  // v: the byte biased by 128
    const int q = a.lut ? (int)a.lut[v] : v - 128;
    from_max[v] = (long long)(q * 256) * (long long)pa.m_max + pa.k;
  }
  __syncthreads();
  grid_dependency_wait();
  grid_dependency_release();
  constexpr int VB = VW == 0 ? 1 : 4 * VW;  // channels per thread
  constexpr int NW = VW == 0 ? 1 : VW;
  const int idx = blockIdx.x * kStripThreads + threadIdx.x;
  if (idx >= threads) return;
  const int strip_of_all = idx / cols, col = idx - strip_of_all * cols;
  const int n = strip_of_all / strips, oh0 = (strip_of_all - n * strips) * strip_rows;
  const int nrows = min(strip_rows, a.OH - oh0);
  const int groups = a.C / VB;
  const int ow = col / groups, g = col - ow * groups;
  const int iw0 = ow * S - a.pad_l, ih0 = oh0 * S - a.pad_t;
  const long long row_bytes = (long long)a.W * a.C;
  const int8_t* px = a.x + (size_t)n * a.H * row_bytes + (long long)ih0 * row_bytes + (long long)iw0 * a.C + g * VB;
  int8_t* out = a.out + (((size_t)n * a.OH + oh0) * a.OW + ow) * a.C + g * VB;
  const bool narrow = pa.clamp_min != -128 || pa.clamp_max != 127;
  const uint32_t lo2 = (uint32_t)(pa.clamp_min & 0xffff) * 0x10001u, hi2 = (uint32_t)(pa.clamp_max & 0xffff) * 0x10001u;
  struct Raw {
    uint32_t w[K][NW];
  };
  // horizontal reductions of one input row: bytes 0 and 2 (e), 1 and 3 (o) of every word, sums (s) and maxima (m)
  struct Row {
    uint32_t se[NW], so[NW], me[NW], mo[NW];
  };
  // EDGE: some window of the warp may hang over the frame
  auto strip = [&](auto edge) {
    constexpr bool EDGE = decltype(edge)::value;
    bool col_ok[K];
    int ncol = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      col_ok[k] = !EDGE || (iw0 + k >= 0 && iw0 + k < a.W);
      ncol += col_ok[k];
    }
    auto load_row = [&](int ih, Raw& r) {
      const bool row_ok = !EDGE || (ih >= 0 && ih < a.H);
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (EDGE) {
#pragma unroll
          for (int j = 0; j < NW; j++) r.w[k][j] = 0x80808080u;  // outside: nothing to the sum, the lowest value to the maximum
        }
        if (row_ok && col_ok[k]) {
          const int8_t* p = px + (size_t)k * a.C;
          if (VW == 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(p);
            r.w[k][0] = v.x; r.w[k][NW > 1 ? 1 : 0] = v.y; r.w[k][NW > 2 ? 2 : 0] = v.z; r.w[k][NW > 3 ? 3 : 0] = v.w;
          } else if (VW == 1) {
            r.w[k][0] = *reinterpret_cast<const uint32_t*>(p);
          } else {
            r.w[k][0] = (uint32_t)(uint8_t)*p;
          }
        }
      }
      px += row_bytes;
    };
    auto reduce = [&](const Raw& raw) {
      Row r;
#pragma unroll
      for (int j = 0; j < NW; j++) {
        uint32_t e[K], o[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
          e[k] = (raw.w[k][j] ^ 0x80808080u) & 0x00ff00ffu;
          o[k] = VW == 0 ? 0u : __byte_perm(raw.w[k][j], 0, 0x4341) ^ 0x00800080u;
        }
        r.se[j] = row_sum<K>(e);
        r.me[j] = max_u16x2_of<K>(e);
        r.so[j] = VW == 0 ? 0u : row_sum<K>(o);
        r.mo[j] = VW == 0 ? 0u : max_u16x2_of<K>(o);
      }
      return r;
    };
    int ih = ih0;
    Row rows[K];  // the window's
    Raw next[S];  // the rows the next step adds, on their way while the last ones are reduced
#pragma unroll
    for (int i = 0; i < K - S; i++) {
      Raw raw;
      load_row(ih++, raw);
      rows[S + i] = reduce(raw);
    }
#pragma unroll
    for (int i = 0; i < S; i++) load_row(ih++, next[i]);
    int4 c = __ldg(a.by_count + K * K);
#pragma unroll 1
    for (int r = 0; r < nrows; r++) {
#pragma unroll
      for (int i = 0; i < K - S; i++) rows[i] = rows[S + i];
#pragma unroll
      for (int i = 0; i < S; i++) rows[K - S + i] = reduce(next[i]);
      if (r + 1 < nrows) {
#pragma unroll
        for (int i = 0; i < S; i++) load_row(ih++, next[i]);
      }
      if (EDGE) {
        const int top = ih0 + r * S;
        c = __ldg(a.by_count + ncol * (min(top + K, a.H) - max(top, 0)));
      }
      const unsigned long long kk = ((unsigned long long)(uint32_t)c.w << 32) | (uint32_t)c.z;
      auto average = [&](uint32_t sum_high) { return (int)(((unsigned long long)sum_high * (uint32_t)c.x + kk) >> 32); };
      uint32_t res[NW];
#pragma unroll
      for (int j = 0; j < NW; j++) {
        uint32_t t[K];
#pragma unroll
        for (int i = 0; i < K; i++) t[i] = rows[i].se[j];
        const uint32_t se = sum_of<K>(t);
#pragma unroll
        for (int i = 0; i < K; i++) t[i] = rows[i].me[j];
        const uint32_t me = max_u16x2_of<K>(t);
#pragma unroll
        for (int i = 0; i < K; i++) t[i] = rows[i].so[j];
        const uint32_t so = sum_of<K>(t);
#pragma unroll
        for (int i = 0; i < K; i++) t[i] = rows[i].mo[j];
        const uint32_t mo = max_u16x2_of<K>(t);
        // the average's bytes in the high byte of 16-bit fields (saturated as the op does), then the linear form
        const uint32_t qe = pack_sat_s16x2(average(se << 16), average(se & 0xffff0000u));
        const int h0 = mad_wide_hi(sx8_shl8<1>(qe), pa.m_avg, from_max[me & 0xffffu]) >> pa.f;
        const int h2 = VW == 0 ? h0 : mad_wide_hi(sx8_shl8<3>(qe), pa.m_avg, from_max[me >> 16]) >> pa.f;
        int h1 = h0, h3 = h0;
        if (VW != 0) {
          const uint32_t qo = pack_sat_s16x2(average(so << 16), average(so & 0xffff0000u));
          h1 = mad_wide_hi(sx8_shl8<1>(qo), pa.m_avg, from_max[mo & 0xffffu]) >> pa.f;
          h3 = mad_wide_hi(sx8_shl8<3>(qo), pa.m_avg, from_max[mo >> 16]) >> pa.f;
        }
        res[j] = narrow ? clamp_pack4(h0, h1, h2, h3, lo2, hi2) : sat_pack4(h0, h1, h2, h3);
      }
      if (VW == 4)
        *reinterpret_cast<uint4*>(out) = make_uint4(res[0], res[NW > 1 ? 1 : 0], res[NW > 2 ? 2 : 0], res[NW > 3 ? 3 : 0]);
      else if (VW == 1) *reinterpret_cast<uint32_t*>(out) = res[0];
      else *out = (int8_t)res[0];
      out += (size_t)a.OW * a.C;
    }
  };
  const bool inside = iw0 >= 0 && iw0 + K <= a.W && ih0 >= 0 && ih0 + (nrows - 1) * S + K <= a.H;
  if (__all_sync(__activemask(), inside)) strip(std::false_type{});
  else strip(std::true_type{});
}


// ---- any other window ----
// I: index type, 32 bits where the tensor allows (a 64-bit division costs more than a window of loads)
template <int VEC, typename I>  // channels per thread: 16 (uint4) or 1
__global__ void __launch_bounds__(kThreads) maxpool_kernel(PoolArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  const int groups = a.C / VEC;
  const I total = (I)a.N * a.OH * a.OW * groups;
  for (I idx = (I)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (I)gridDim.x * blockDim.x) {
    int g = (int)(idx % groups);
    I p = idx / groups;
    int ow = (int)(p % a.OW);
    I t = p / a.OW;
    int oh = (int)(t % a.OH);
    int n = (int)(t / a.OH);
    const int8_t* xin = a.x + (size_t)n * a.H * a.W * a.C + g * VEC;
    if (VEC == 16) {
      uint32_t best[4] = {0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u};
      const uint32_t padw = (uint32_t)(a.pad_value & 0xff) * 0x01010101u;
      for (int kh = 0; kh < a.KH; kh++) {
        int ih = oh * a.stride_h - a.pad_t + kh;
        for (int kw = 0; kw < a.KW; kw++) {
          int iw = ow * a.stride_w - a.pad_l + kw;
          uint4 v;
          if (ih < 0 || ih >= a.H || iw < 0 || iw >= a.W) v = make_uint4(padw, padw, padw, padw);
          else v = *reinterpret_cast<const uint4*>(xin + ((size_t)ih * a.W + iw) * a.C);
          best[0] = __vmaxs4(best[0], v.x);
          best[1] = __vmaxs4(best[1], v.y);
          best[2] = __vmaxs4(best[2], v.z);
          best[3] = __vmaxs4(best[3], v.w);
        }
      }
      *reinterpret_cast<uint4*>(a.out + (size_t)p * a.C + g * 16) = make_uint4(best[0], best[1], best[2], best[3]);
    } else {
      int best = -128;
      for (int kh = 0; kh < a.KH; kh++) {
        int ih = oh * a.stride_h - a.pad_t + kh;
        for (int kw = 0; kw < a.KW; kw++) {
          int iw = ow * a.stride_w - a.pad_l + kw;
          int v = (ih < 0 || ih >= a.H || iw < 0 || iw >= a.W) ? a.pad_value
                                                               : (int)xin[((size_t)ih * a.W + iw) * a.C];
          best = max(best, v);
        }
      }
      a.out[(size_t)p * a.C + g] = (int8_t)best;
    }
  }
}

// The same on int16 tensors (the reference's MaxPool2D i16 -> i16): 8 channels per thread, or 1.
template <int VEC, typename I>
__global__ void __launch_bounds__(kThreads) maxpool_i16_kernel(PoolArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  const int16_t* x = reinterpret_cast<const int16_t*>(a.x);
  int16_t* out = reinterpret_cast<int16_t*>(a.out);
  const int groups = a.C / VEC;
  const I total = (I)a.N * a.OH * a.OW * groups;
  for (I idx = (I)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (I)gridDim.x * blockDim.x) {
    const int g = (int)(idx % groups);
    const I p = idx / groups;
    const int ow = (int)(p % a.OW);
    const I t = p / a.OW;
    const int oh = (int)(t % a.OH);
    const int n = (int)(t / a.OH);
    const int16_t* xin = x + (size_t)n * a.H * a.W * a.C + g * VEC;
    if (VEC == 8) {
      uint32_t best[4] = {0x80008000u, 0x80008000u, 0x80008000u, 0x80008000u};
      const uint32_t padw = (uint32_t)(a.pad_value & 0xffff) * 0x00010001u;
      for (int kh = 0; kh < a.KH; kh++) {
        const int ih = oh * a.stride_h - a.pad_t + kh;
        for (int kw = 0; kw < a.KW; kw++) {
          const int iw = ow * a.stride_w - a.pad_l + kw;
          uint4 v;
          if (ih < 0 || ih >= a.H || iw < 0 || iw >= a.W) v = make_uint4(padw, padw, padw, padw);
          else v = *reinterpret_cast<const uint4*>(xin + ((size_t)ih * a.W + iw) * a.C);
          best[0] = __vmaxs2(best[0], v.x);
          best[1] = __vmaxs2(best[1], v.y);
          best[2] = __vmaxs2(best[2], v.z);
          best[3] = __vmaxs2(best[3], v.w);
        }
      }
      *reinterpret_cast<uint4*>(out + (size_t)p * a.C + g * 8) = make_uint4(best[0], best[1], best[2], best[3]);
    } else {
      int best = -32768;
      for (int kh = 0; kh < a.KH; kh++) {
        const int ih = oh * a.stride_h - a.pad_t + kh;
        for (int kw = 0; kw < a.KW; kw++) {
          const int iw = ow * a.stride_w - a.pad_l + kw;
          const int v = (ih < 0 || ih >= a.H || iw < 0 || iw >= a.W) ? a.pad_value : (int)xin[((size_t)ih * a.W + iw) * a.C];
          best = max(best, v);
        }
      }
      out[(size_t)p * a.C + g] = (int16_t)best;
    }
  }
}

// reciprocal_scale of the TOSA spec (compiler/torq/Conversions/TosaToTorqHL/Patterns.cpp:796-805)
__device__ __forceinline__ void reciprocal_scale(uint32_t count, int32_t& mult, int32_t& shift) {
  int k = 32 - __clz((int)(count - 1));
  if (count == 1) k = 0;
  long long numerator = ((1ll << 30) + 1) << k;
  mult = (int32_t)(numerator / (long long)count);
  shift = 30 + k;
}

// ---- average pool: tosa.avg_pool2d acc_type=i32; count excludes padding ----
// The rescale depends only on the number of taps inside the image, so the block fills a table indexed by that
// count once (one 64-bit division per entry instead of one per output). Entry {M, 2^(S-30), S-29, count}:
// TOSA's (v * M + 2^(S-1)) >> S with S = 30 + k >= 30 equals (8v * M + 2^(S+2)) >> (S + 3), and since the constant
// has a zero low word that is (mulhi(8v, M) + 2^(S-30)) >> (S - 29): exact, 32-bit.
constexpr int kAvgMaxTaps = 256;
template <int VEC, typename I>  // 16, 4 or 1 channels per thread
__global__ void __launch_bounds__(kThreads) avgpool_kernel(PoolArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ int4 by_count[kAvgMaxTaps + 1];
  for (int c = threadIdx.x; c <= a.KH * a.KW; c += blockDim.x) {
    int32_t mult, shift;
    reciprocal_scale(c ? (uint32_t)c : 1u, mult, shift);
    by_count[c] = make_int4(mult, 1 << (shift - 30), shift - 29, c);
  }
  __syncthreads();
  const int groups = a.C / VEC;
  const I total = (I)a.N * a.OH * a.OW * groups;
  for (I idx = (I)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (I)gridDim.x * blockDim.x) {
    int g = (int)(idx % groups);
    I p = idx / groups;
    int ow = (int)(p % a.OW);
    I t = p / a.OW;
    int oh = (int)(t % a.OH);
    int n = (int)(t / a.OH);
    const int8_t* xin = a.x + (size_t)n * a.H * a.W * a.C + g * VEC;
    int acc[VEC];
#pragma unroll
    for (int j = 0; j < VEC; j++) acc[j] = 0;
    int count = 0;
    for (int kh = 0; kh < a.KH; kh++) {
      int ih = oh * a.stride_h - a.pad_t + kh;
      if (ih < 0 || ih >= a.H) continue;
      for (int kw = 0; kw < a.KW; kw++) {
        int iw = ow * a.stride_w - a.pad_l + kw;
        if (iw < 0 || iw >= a.W) continue;
        count++;
        const int8_t* px = xin + ((size_t)ih * a.W + iw) * a.C;
        if (VEC == 16) {
          const uint4 v = *reinterpret_cast<const uint4*>(px);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 16; j++) acc[j] = __dp4a((int)w[j >> 2], 1 << (8 * (j & 3)), acc[j]);  // adds byte j, sign-extended
        } else if (VEC == 4) {
          const uint32_t v = *reinterpret_cast<const uint32_t*>(px);
#pragma unroll
          for (int j = 0; j < 4; j++) acc[j] = __dp4a((int)v, 1 << (8 * j), acc[j]);
        } else {
          acc[0] += (int)px[0];
        }
      }
    }
    const int4 k = by_count[count];
    const int zsum = count * a.input_zp;
    int q[VEC];
#pragma unroll
    for (int j = 0; j < VEC; j++) {
      const int r = ((__mulhi((acc[j] - zsum) * 8, k.x) + k.y) >> k.z) + a.output_zp;
      q[j] = max(-128, min(127, r));
    }
    if (VEC == 16)
      *reinterpret_cast<uint4*>(a.out + (size_t)p * a.C + g * 16) =
          make_uint4(pack4(q[0], q[1], q[2], q[3]), pack4(q[4], q[5], q[6], q[7]), pack4(q[8], q[9], q[10], q[11]),
                     pack4(q[12], q[13], q[14], q[15]));
    else if (VEC == 4) *reinterpret_cast<uint32_t*>(a.out + (size_t)p * a.C + g * 4) = pack4(q[0], q[1], q[2], q[3]);
    else a.out[(size_t)p * a.C + g] = (int8_t)q[0];
  }
}

// Large windows over few outputs (the global pool at the end of a classifier: 7x7 -> 1x1): a warp per output pixel
// and group of 16 channels, the taps spread over the lanes, sums combined by shuffles. Same arithmetic as above.
__global__ void __launch_bounds__(kThreads) avgpool_warp_kernel(PoolArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ int4 by_count[kAvgMaxTaps + 1];
  for (int c = threadIdx.x; c <= a.KH * a.KW; c += blockDim.x) {
    int32_t mult, shift;
    reciprocal_scale(c ? (uint32_t)c : 1u, mult, shift);
    by_count[c] = make_int4(mult, 1 << (shift - 30), shift - 29, c);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int groups = a.C / 16;
  const long long total = (long long)a.N * a.OH * a.OW * groups;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int taps = a.KH * a.KW;
  for (long long idx = warp0; idx < total; idx += nwarps) {
    const int g = (int)(idx % groups);
    const long long p = idx / groups;
    const int ow = (int)(p % a.OW);
    const long long t = p / a.OW;
    const int oh = (int)(t % a.OH);
    const int n = (int)(t / a.OH);
    const int8_t* xin = a.x + (size_t)n * a.H * a.W * a.C + g * 16;
    int acc[16];
#pragma unroll
    for (int j = 0; j < 16; j++) acc[j] = 0;
    int count = 0;
    for (int tap = lane; tap < taps; tap += 32) {
      const int kh = tap / a.KW, kw = tap - kh * a.KW;
      const int ih = oh * a.stride_h - a.pad_t + kh, iw = ow * a.stride_w - a.pad_l + kw;
      if (ih < 0 || ih >= a.H || iw < 0 || iw >= a.W) continue;
      count++;
      const uint4 v = *reinterpret_cast<const uint4*>(xin + ((size_t)ih * a.W + iw) * a.C);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 16; j++) acc[j] = __dp4a((int)w[j >> 2], 1 << (8 * (j & 3)), acc[j]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      count += __shfl_xor_sync(0xffffffffu, count, o);
#pragma unroll
      for (int j = 0; j < 16; j++) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    if (lane == 0) {
      const int4 k = by_count[count];
      const int zsum = count * a.input_zp;
      int q[16];
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const int r = ((__mulhi((acc[j] - zsum) * 8, k.x) + k.y) >> k.z) + a.output_zp;
        q[j] = max(-128, min(127, r));
      }
      *reinterpret_cast<uint4*>(a.out + (size_t)p * a.C + g * 16) =
          make_uint4(pack4(q[0], q[1], q[2], q[3]), pack4(q[4], q[5], q[6], q[7]), pack4(q[8], q[9], q[10], q[11]),
                     pack4(q[12], q[13], q[14], q[15]));
    }
  }
}


}  // namespace

bool pool_strip_applies(const PoolArgs& a) {
  if (a.elem16 || a.KH != a.KW || a.stride_h != a.stride_w || a.N > 65535 || a.OH > 65535) return false;
  const int k = a.KH, s = a.stride_h;
  return (k == 2 && s == 2) || (k == 3 && (s == 1 || s == 2)) || (k == 5 && s == 1);
}

bool pool_avg_records(int taps, int input_zp, int output_zp, std::vector<int4>& out) {
  out.assign((size_t)taps + 1, make_int4(0, 0, 0, 0));
  for (int c = 1; c <= taps; c++) {
    // reciprocal_scale of the TOSA spec, as on the device
    int k = 0;
    while (k < 32 && ((uint32_t)(c - 1) >> k) != 0) k++;
    const long long numerator = ((1ll << 30) + 1) << k;
    const long long mult = numerator / c;
    const int shift = 30 + k;
    // (v * 2^16) * m / 2^40 ~ v / c. TOSA's factor is a trace above 1 / c, so ties round away from zero on both sides; the
    // slope has to be a trace above it too for one K to serve both
    const unsigned long long m = (((unsigned long long)mult << 24) >> shift) + 1;
    long long lo = INT64_MIN, hi = INT64_MAX;  // K with lo <= K <= hi gives TOSA's result for every sum of c biased bytes
    for (int v = 0; v <= 255 * c; v++) {
      const long long sum = (long long)v - 128ll * c - (long long)c * input_zp;
      const long long r = (long long)(int32_t)((sum * mult + (1ll << (shift - 1))) >> shift) + output_zp;
      const long long q = (long long)((unsigned long long)v << 16) * (long long)m;
      if (r > -128) lo = std::max(lo, ((r < 127 ? r : 127) << 40) - q);
      if (r < 127) hi = std::min(hi, (((r > -128 ? r : -128) + 1) << 40) - q - 1);
    }
    if (lo > hi) return false;
    const long long kk = lo == INT64_MIN ? hi : hi == INT64_MAX ? lo : lo + (hi - lo) / 2;
    out[c] = make_int4((int)(uint32_t)m, 0, (int)(uint32_t)kk, (int)(kk >> 32));
  }
  return true;
}

namespace {
template <int VW, int K, int S, int ROWS, bool AVG>
void launch_strip(const PoolArgs& a, cudaStream_t stream) {
  const int vb = VW == 0 ? 1 : 4 * VW;
  const long long cols = (long long)a.OW * (a.C / vb);
  const dim3 grid((unsigned)((cols + kStripThreads - 1) / kStripThreads), (unsigned)((a.OH + ROWS - 1) / ROWS), (unsigned)a.N);
  if (a.lut) launch_dependent(pool_strip_kernel<VW, K, S, ROWS, AVG, true>, grid, dim3(kStripThreads), 0, stream, a);
  else launch_dependent(pool_strip_kernel<VW, K, S, ROWS, AVG, false>, grid, dim3(kStripThreads), 0, stream, a);
}
// How much one thread does. Long strips and 16 channels cost the fewest loads per output; a small frame is bound by the
// latency of a thread's own chain instead, so the work is cut finer until about 512 threads per SM exist.
template <int K, int S, bool AVG>
void launch_strip_shape(const PoolArgs& a, cudaStream_t stream) {
  const bool al = (((uintptr_t)a.x | (uintptr_t)a.out) & 15) == 0;
  const long long pixels = (long long)a.N * a.OH * a.OW, want = 148ll * 512;
  if (al && (a.C & 15) == 0 && pixels * (a.C / 16) >= 4 * want) launch_strip<4, K, S, 4, AVG>(a, stream);
  else if (al && (a.C & 15) == 0 && pixels * (a.C / 16) >= want) launch_strip<4, K, S, 1, AVG>(a, stream);
  else if ((a.C & 3) == 0 && pixels * (a.C / 4) >= 4 * want) launch_strip<1, K, S, 4, AVG>(a, stream);
  else if ((a.C & 3) == 0) launch_strip<1, K, S, 1, AVG>(a, stream);
  else launch_strip<0, K, S, 4, AVG>(a, stream);
}
template <bool AVG>
bool try_strip(const PoolArgs& a, cudaStream_t stream) {
  if (!pool_strip_applies(a) || (AVG && !a.by_count)) return false;
  if (a.KH == 2) launch_strip_shape<2, 2, AVG>(a, stream);
  else if (a.KH == 3 && a.stride_h == 1) launch_strip_shape<3, 1, AVG>(a, stream);
  else if (a.KH == 3) launch_strip_shape<3, 2, AVG>(a, stream);
  else launch_strip_shape<5, 1, AVG>(a, stream);
  return true;
}
bool fits32(const PoolArgs& a) { return (long long)a.N * a.OH * a.OW * a.C < (1ll << 30); }

template <int VW, int K, int S>
cudaError_t launch_pool_add_strips(const PoolAddArgs& a, int rows, cudaStream_t stream) {
  const int vb = VW == 0 ? 1 : 4 * VW, cols = a.pool.OW * (a.pool.C / vb), strips = (a.pool.OH + rows - 1) / rows;
  const int threads = a.pool.N * strips * cols;  // pool_add_applies: fits
  return launch_dependent(pool_add_kernel<VW, K, S>, dim3((unsigned)((threads + kStripThreads - 1) / kStripThreads)), dim3(kStripThreads), 0,
                          stream, a, cols, strips, rows, threads);
}
// As in launch_strip_shape, and the strip shortened step by step: two rows halve what a warp has to do in turn at the cost of a quarter
// more input rows. Words of 4 channels take strips of 8 where there is work for them (27.3 -> 23.8 us at the size above).
template <int K, int S>
cudaError_t launch_pool_add_shape(const PoolAddArgs& pa, cudaStream_t stream) {
  const PoolArgs& a = pa.pool;
  const uintptr_t at = (uintptr_t)a.x | (uintptr_t)a.out;
  const long long pixels = (long long)a.N * a.OH * a.OW, want = 512ll * current_sm_count(), wide = pixels * (a.C / 16) / want, words = pixels * (a.C / 4) / want;
  if ((at & 15) == 0 && (a.C & 15) == 0 && wide >= 1) return launch_pool_add_strips<4, K, S>(pa, wide >= 4 ? 4 : wide >= 2 ? 2 : 1, stream);
  if ((at & 3) == 0 && (a.C & 3) == 0) return launch_pool_add_strips<1, K, S>(pa, words >= 8 ? 8 : words >= 4 ? 4 : 1, stream);
  return launch_pool_add_strips<0, K, S>(pa, 4, stream);
}
}  // namespace

bool pool_add_applies(const PoolArgs& a) {
  return pool_strip_applies(a) && a.pad_value == -128 && (long long)a.N * a.OH * a.OW * a.C < (1ll << 31) - kStripThreads;
}

cudaError_t launch_pool_add(const PoolAddArgs& a, cudaStream_t stream) {
  if (a.pool.KH == 2) return launch_pool_add_shape<2, 2>(a, stream);
  if (a.pool.KH == 5) return launch_pool_add_shape<5, 1>(a, stream);
  return a.pool.stride_h == 1 ? launch_pool_add_shape<3, 1>(a, stream) : launch_pool_add_shape<3, 2>(a, stream);
}

void launch_maxpool(const PoolArgs& a, cudaStream_t stream) {
  if (try_strip<false>(a, stream)) return;
  const long long pixels = (long long)a.N * a.OH * a.OW;
  const bool small = fits32(a);
  auto go = [&](auto k32, auto k64, int vec) {
    const dim3 grid(grid_for(pixels * (a.C / vec)));
    if (small) launch_dependent(k32, grid, dim3(kThreads), 0, stream, a);
    else launch_dependent(k64, grid, dim3(kThreads), 0, stream, a);
  };
  if (a.elem16) {
    if ((a.C & 7) == 0) go(maxpool_i16_kernel<8, unsigned>, maxpool_i16_kernel<8, long long>, 8);
    else go(maxpool_i16_kernel<1, unsigned>, maxpool_i16_kernel<1, long long>, 1);
    return;
  }
  if ((a.C & 15) == 0) go(maxpool_kernel<16, unsigned>, maxpool_kernel<16, long long>, 16);
  else go(maxpool_kernel<1, unsigned>, maxpool_kernel<1, long long>, 1);
}

void launch_avgpool(const PoolArgs& a, cudaStream_t stream) {
  if (try_strip<true>(a, stream)) return;
  const long long pixels = (long long)a.N * a.OH * a.OW;
  const bool small = fits32(a);
  auto go = [&](auto k32, auto k64, int vec) {
    const dim3 grid(grid_for(pixels * (a.C / vec)));
    if (small) launch_dependent(k32, grid, dim3(kThreads), 0, stream, a);
    else launch_dependent(k64, grid, dim3(kThreads), 0, stream, a);
  };
  if ((a.C & 15) == 0 && ((uintptr_t)a.x & 15) == 0 && ((uintptr_t)a.out & 15) == 0) {
    const long long total = pixels * (a.C / 16);
    // few outputs with many taps each: spread the taps over a warp
    if (a.KH * a.KW >= 16 && total < 148ll * 2048) launch_dependent(avgpool_warp_kernel, dim3(grid_for(total * 32)), dim3(kThreads), 0, stream, a);
    else go(avgpool_kernel<16, unsigned>, avgpool_kernel<16, long long>, 16);
  } else if ((a.C & 3) == 0) {
    go(avgpool_kernel<4, unsigned>, avgpool_kernel<4, long long>, 4);
  } else {
    go(avgpool_kernel<1, unsigned>, avgpool_kernel<1, long long>, 1);
  }
}

}  // namespace tb200
