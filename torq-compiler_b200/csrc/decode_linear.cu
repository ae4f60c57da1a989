// The products and the attention of a decode step run op by op: int8 weights on bf16 activations of up to 32 tokens, and one
// query per sequence against its cache. Every one of them moves a few MB, a microsecond or two of HBM time, so what bounds a
// step is how early the bytes are asked for and how few launches stand in a row:
//   * each kernel asks for its weights (or cache lines) before it waits for the kernel ahead of it: the weights belong to
//     the program, so they stream in while the activations are still being made;
//   * a long K is split over the warps of a block and, where the activations would not fit shared memory, over the blocks of
//     a cluster; the fp32 sums meet in shared memory (the cluster's through distributed shared memory), in one fixed order,
//     and the finished bf16 values leave the kernel - no partial sums in global memory;
//   * the op behind a product runs in its epilogue where a block holds what it needs: GeGLU (a warp's tile is 16 gate rows
//     and the 16 matching up rows), head norm + RoPE + cache append (a cluster of eight blocks holds a head), the arg max
//     over the logits.
//   * weights are in L2 before their kernel starts: a product asks for those of the product after the next one (blocks that a small grid leaves
//     out do it, else every thread a line or two);
//   * up to two sequences the norms in front of the q/k/v and the gate/up product run in it: every block norms the rows for itself, which costs
//     less than a launch whose result it would have to wait for.
// Measured at the Gemma-3-1B shape at position 1024, launches serialised, us per launch (split-K kernels of decoder.cu, 32 sequences)
// -> here with 32 / one sequence (one sequence: with their norms): attention 10.6 + 3.4 -> 9.2 / 6.3, gate/up + GeGLU 10.5 + 4.4 -> 11.1 /
// 7.9, norms 8.6 -> 2.4, LM head 125 -> 94.5 / 50.3, arg max 24 -> 2.3; q/k/v + head norm + RoPE 8.8 / 7.5, o and down 7.5 / 5.2 on average. A
// whole step, launches overlapping: 1.13 / 0.67 ms. What the last steps gave when they were made, one sequence: 0.81 -> 0.75 ms by norms that
// release before their wait, 0.75 -> 0.70 by norms inside products, 0.01 by the later product's weights.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "dependent_launch.cuh"
#include "device_memory.cuh"
#include "kernels.h"
#include "linear_shape.h"

namespace tb200 {
namespace {

__device__ __forceinline__ float bf2f(uint16_t v) { return __uint_as_float((uint32_t)v << 16); }
__device__ __forceinline__ uint16_t f2bf(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }
__device__ __forceinline__ float rbf(float f) { return bf2f(f2bf(f)); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
// into a float of another block of the cluster, at the address the same float has in this block
__device__ __forceinline__ void st_peer(uint32_t addr, int rank, float v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 2^n, n in [-126, 127]
__device__ __forceinline__ float pow2(int n) { return __int_as_float((n + 127) << 23); }
// Four signed bytes -> bf16 pairs (k, k+1) and (k+2, k+3), exact. 0x4300 | u is 128 + u for the seven low bits, and the top
// bit turns the 128 that is taken off again into 256.
__device__ __forceinline__ void s8x4_to_bf16x4(uint32_t w, uint32_t& lo, uint32_t& hi) {
  const uint32_t p = __byte_perm(w, 0x43434343u, 0x4140), q = __byte_perm(w, 0x43434343u, 0x4342);
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(lo) : "r"(p & 0xff7fff7fu), "r"(p & 0xff80ff80u));
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(hi) : "r"(q & 0xff7fff7fu), "r"(q & 0xff80ff80u));
}
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * x * (1.0f + tanhf(k0 * (x + k1 * x * x * x)));
}

// ---------------------------------------------------------------------------------------------------------------
// y[b, n] = sum_k x[b, k] * W[n, k] * scale[n]: weights are the 16-row operand of mma.sync m16n8k16 (bf16, fp32
// accumulation), tokens the 8-column one. A warp works on a tile of 32 weight rows (each activation fragment read from shared
// memory then serves two instructions: at 32 tokens these reads bounded a 16-row tile) and one of TK groups of 64-byte
// blocks of K, whose weights it copies into a ring of its own (cp.async; nothing but the warp itself waits for them). The
// activations of the block's K range are staged once per block. TK depends on N and K alone, and a result is the sum of its
// TK groups in order, so it does not depend on the mode or on how groups are spread over warps and blocks (fp32 results that SLICED
// takes are the exception, whatever stands behind them).
//   kStore: bf16 or fp32 results.                      kGeglu: bf16(bf16(gelu(gate)) * up), tiles of 16 gate and 16 up rows.
//   kRope:  a cluster of eight blocks is one head of 256: head norm, RoPE, q out / cache append (arithmetic of rope_kv_kernel).
//   kStream: one group and a warp per tile, blocks stay and walk the tiles (the LM head); fp32 or bf16 results and, with
//            cand_v, the block's arg-max candidates per token. SLICED (fp32 results of up to eight tokens): int8 instructions on the weights as they are and
//            on four int8 slices of every activation, exact integer sums joined in fp32. The conversion of weights to bf16 was what bounded it:
//            302 MB of weights for one token 62.2 -> 49.1 us (46 us of HBM time), against 64 bits the error falls from 1.2e-7 to 0.3e-7.
//            Tokens whose row four slices do not hold exactly go through the weights once more in bf16.
// ---------------------------------------------------------------------------------------------------------------

constexpr int kNoSlices = 0x7fffffff;  // in place of a shift: four slices do not hold the token's activations exactly

template <int NT, int MODE, bool SLICED>
__global__ void __launch_bounds__(512, 1) linear_w8_kernel(const LinearArgs a) {
  extern __shared__ __align__(128) unsigned char sm[];
  // blocks beyond the product's own bring a later product's weights to L2
  auto prefetch = [&](int block, int count) {
    for (uint32_t at = (block * blockDim.x + threadIdx.x) * 128u; at < a.next_bytes; at += count * blockDim.x * 128u)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a.next + at));
  };
  if (MODE != kStream && (int)blockIdx.x >= a.work_blocks) {
    prefetch(blockIdx.x - a.work_blocks, gridDim.x - a.work_blocks);
    return;
  }
  const int kg_log2 = __ffs(a.kg) - 1, ck_log2 = __ffs(a.ck) - 1, tk_log2 = kg_log2 + ck_log2;  // all powers of two
  const int rank = blockIdx.x & (a.ck - 1);  // K slice of this block (clusters are consecutive blocks)
  const int row_block = blockIdx.x >> ck_log2;
  const int blocks = a.K / kBlk;
  const int kb0 = blocks * (rank << kg_log2) >> tk_log2, kb1 = blocks * ((rank + 1) << kg_log2) >> tk_log2;  // K blocks of this thread block
  constexpr int kTok = SLICED ? 8 : NT * 8, kPitch = kTok + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const int kg = warp & (a.kg - 1), rt = warp >> kg_log2;
  const int group = (rank << kg_log2) + kg;
  const int wb0 = blocks * group >> tk_log2, nb = (blocks * (group + 1) >> tk_log2) - wb0;  // and of this warp
  const int tile0 = MODE == kStream ? blockIdx.x * a.rt + rt : row_block * a.rt + rt;
  const int tile_step = gridDim.x * a.rt;
  const int tiles = (MODE == kStream) ? (tile0 < a.tiles ? (a.tiles - tile0 + tile_step - 1) / tile_step : 0) : tile0 < a.tiles ? 1 : 0;
  const int total = tiles * nb;
  const uint32_t x_addr = smem_u32(sm), ring = x_addr + (uint32_t)a.x_bytes + (uint32_t)(warp * a.stages) * kStageBytes;

  // ---- weights: this warp's first blocks, before anything else ----
  auto weight_row = [&](int tile, int r) { return MODE == kGeglu ? (r < 16 ? tile * 16 + r : a.N / 2 + tile * 16 + r - 16) : tile * kTileRows + r; };
  auto row_valid = [&](int tile, int r) { return MODE == kGeglu ? tile * 16 + (r & 15) < a.N / 2 : tile * kTileRows + r < a.N; };
  int is_tile = tile0, is_kb = 0, is_stage = 0;
  auto issue = [&]() {
    // lane -> 16-byte piece tig of rows g, g + 8, g + 16, g + 24
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int r = g + 8 * j;
      const bool v = row_valid(is_tile, r);
      cp_async16(ring + is_stage * kStageBytes + r * kBlk + tig * 16, a.W + (v ? (size_t)weight_row(is_tile, r) * a.K : 0) + (size_t)(wb0 + is_kb) * kBlk + tig * 16, v);
    }
    if (++is_kb == nb) { is_kb = 0; is_tile += tile_step; }
    if (++is_stage == a.stages) is_stage = 0;
  };
  int issued = 0;
  for (; issued < a.stages && issued < total; issued++) {
    issue();
    cp_commit();
  }
  if (MODE != kStream && a.next_bytes && gridDim.x == a.work_blocks) prefetch(blockIdx.x, gridDim.x);
  if (SLICED && MODE == kStream)  // the loop below counts groups
    for (int j = issued; j < kStreamStages; j++) cp_commit();
  // (constants stay raw until they are used: a conversion here would wait for HBM before the activations are even asked for)
  float rope_c = 0.f, rope_s = 0.f;
  uint16_t norm_w = 0, norm_w_other = 0;
  int pos = 0;
  const int head = MODE == kRope ? blockIdx.x / 8 : 0, part = MODE == kRope ? blockIdx.x % 8 : 0;
  auto rope_angle = [&](int p) {  // the position's rotation for this lane's row
    pos = p < 0 ? 0 : (p >= a.T ? a.T - 1 : p);
    const int i = (part & 3) * 32 + lane;
    const float inv_freq = powf(a.theta, -(float)i / 128.0f);
    sincosf((float)pos * inv_freq, &rope_s, &rope_c);
  };
  const bool is_q = head < a.n_q, is_k = head == a.n_q;
  if (MODE == kRope) {
    if (is_q || is_k) {
      const uint16_t* w = (is_q ? a.qw : a.kw) + lane;
      norm_w = __ldg(w + part * 32);
      norm_w_other = __ldg(w + (part ^ 4) * 32);
    }
  }
  // the scales of the block's rows, read once per step and so always from HBM: stored behind the staging
  float* scale_s = reinterpret_cast<float*>(sm + a.scale_off);
  uint16_t scale_r = 0;
  if (MODE != kStream && (int)threadIdx.x < a.rt * kTileRows) {  // never more rows than threads
    const int t = row_block * a.rt + (int)threadIdx.x / kTileRows;
    if (row_valid(t, threadIdx.x % kTileRows)) scale_r = __ldg(a.scale + weight_row(t, threadIdx.x % kTileRows));
  }
  // the norm in front: a thread holds four elements of a row, as in rmsnorm_row_kernel
  constexpr bool kNorm = NT == 1 && (MODE == kGeglu || MODE == kRope);
  const int norm_at = 4 * threadIdx.x;
  uint2 norm_wv = make_uint2(0, 0), norm_wv2 = norm_wv;
  if (kNorm && a.norm_x && norm_at < a.K) {
    norm_wv = __ldg(reinterpret_cast<const uint2*>(a.norm_w + norm_at));
    if (a.norm_w2) norm_wv2 = __ldg(reinterpret_cast<const uint2*>(a.norm_w2 + norm_at));
  }
  if (SLICED)  // zeros in the columns of no token
    for (int col = a.B * kSlices; col < NT * 8; col++)
      for (int i = threadIdx.x; i < blocks * (kBlk / 16); i += blockDim.x) *reinterpret_cast<uint4*>(sm + col * a.x_pitch + 16 * i) = make_uint4(0, 0, 0, 0);
  int pos_seen = 0;
  if (MODE == kRope) {
    pos_seen = __ldcg(a.pos);  // read again behind the wait, and nearly always the same
    rope_angle(pos_seen);
  }
  // Waited for before the first remote store: it says that the block runs, not how far it is, so a peer may only store into
  // memory that nothing else of the block uses (recv_off).
  if (MODE == kRope || a.ck > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  grid_dependency_wait();
  grid_dependency_release();

  // ---- activations of K blocks [kb0, kb1); tokens beyond B read as zero ----
  int* const shifts = reinterpret_cast<int*>(sm + a.side_off);
  int pos_now = pos_seen;
  if (MODE == kRope) pos_now = __ldcg(a.pos);
  const int warps = blockDim.x >> 5;
  if constexpr (SLICED) {
    // A warp slices a token: x = d0 + 2^8 d1 + 2^16 d2 + 2^24 d3 in units of 2^-shift, the largest of the row just below 2^30, digits in
    // [-128, 127]. Exact where no value's exponent but a zero's is more than 22 below the largest one's. A smaller value would lose bits that
    // an fp32 sum keeps (all that is left of the sum where the large ones meet zero weights), so such a row is left to the bf16 form, as one
    // with an infinity or a NaN is. Of rows of 1152 normal values one in 2300 goes there.
    constexpr int kHold = 10;  // 128 values each, kept between the two passes over them
    for (int b = warp; b < a.B; b += warps) {
      const uint16_t* src = a.x + (size_t)b * a.K + 4 * lane;
      auto load = [&](int i) { return 128 * i + 4 * lane < a.K ? __ldcg(reinterpret_cast<const uint2*>(src + 128 * i)) : make_uint2(0, 0); };
      uint2 hold[kHold];
      uint32_t top = 0, low = 0xffffffffu;  // largest magnitude, as bits, and the smallest that is not zero, less one
      auto widen = [&](const uint2& u) {
        top = __vmaxu2(top, u.x & 0x7fff7fffu);
        top = __vmaxu2(top, u.y & 0x7fff7fffu);
        low = __vminu2(low, __vsub2(u.x & 0x7fff7fffu, 0x00010001u));  // (a zero becomes the largest)
        low = __vminu2(low, __vsub2(u.y & 0x7fff7fffu, 0x00010001u));
      };
#pragma unroll
      for (int i = 0; i < kHold; i++) hold[i] = load(i);
#pragma unroll
      for (int i = 0; i < kHold; i++) widen(hold[i]);
      for (int i = kHold; 128 * i < a.K; i++) widen(load(i));
      const uint32_t e = __reduce_max_sync(0xffffffffu, max(top >> 16, top & 0xffffu)) >> 7;  // its exponent, biased
      const uint32_t least = __reduce_min_sync(0xffffffffu, min(low >> 16, low & 0xffffu));
      const int shift = 29 + 127 - max((int)e, 1), first = min(shift, 126);
      // the seven bits behind the smallest one's exponent end at or above a unit (a row of zeros has no smallest one)
      const bool exact = e != 255 && (least == 0xffffu || max((int)e, 1) - max((int)((least + 1) >> 7), 1) <= 22);
      if (lane == 0) shifts[b] = exact ? shift : kNoSlices;
      const float s0 = pow2(first), s1 = pow2(shift - first);
      const uint32_t dst = x_addr + (uint32_t)(b * kSlices * a.x_pitch + 4 * lane);
      auto slice = [&](const uint2& u, int i) {
        uint32_t d[4];
        const uint32_t half[2] = {u.x, u.y};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float x = __uint_as_float(j & 1 ? half[j >> 1] & 0xffff0000u : half[j >> 1] << 16);
          d[j] = ((uint32_t)__float2int_rn(x * s0 * s1) + 0x00808080u) ^ 0x00808080u;  // bytes: the digits
        }
        if (128 * i + 4 * lane >= a.K) return;
        const uint32_t p = __byte_perm(d[0], d[1], 0x5140), q = __byte_perm(d[2], d[3], 0x5140), r = __byte_perm(d[0], d[1], 0x7362), t = __byte_perm(d[2], d[3], 0x7362);
        const uint32_t digit[4] = {__byte_perm(p, q, 0x5410), __byte_perm(p, q, 0x7632), __byte_perm(r, t, 0x5410), __byte_perm(r, t, 0x7632)};
#pragma unroll
        for (int j = 0; j < 4; j++) asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + j * a.x_pitch + 128 * i), "r"(digit[j]) : "memory");
      };
#pragma unroll
      for (int i = 0; i < kHold; i++)
        if (128 * i < a.K) slice(hold[i], i);
      for (int i = kHold; 128 * i < a.K; i++) slice(load(i), i);
    }
    cp_wait<kStreamStages - 1>();
  } else {
    bool staged = false;
    if constexpr (kNorm) {
      if (a.norm_x) {
        staged = true;
        float* red = reinterpret_cast<float*>(sm + a.side_off);  // sums of the two reductions: [row][pass][warp]
        const int norm_warps = (a.K / 4 + 31) / 32;
        float v[kNormTokens][4], r[kNormTokens][4];
        auto four = [](const uint2& u, float (&f)[4]) {
          f[0] = __uint_as_float(u.x << 16);
          f[1] = __uint_as_float(u.x & 0xffff0000u);
          f[2] = __uint_as_float(u.y << 16);
          f[3] = __uint_as_float(u.y & 0xffff0000u);
        };
#pragma unroll
        for (int b = 0; b < kNormTokens; b++) {
          uint2 u = make_uint2(0, 0), ur = u;
          if (b < a.B && norm_at < a.K) {
            u = __ldcg(reinterpret_cast<const uint2*>(a.norm_x + (size_t)b * a.K + norm_at));
            if (a.norm_res) ur = __ldcg(reinterpret_cast<const uint2*>(a.norm_res + (size_t)b * a.K + norm_at));
          }
          four(u, v[b]);
          four(ur, r[b]);
        }
        for (int b = a.B + warp; b < kTok; b += warps)  // no token
          for (int c = lane; c < a.K / 8; c += 32) *reinterpret_cast<uint4*>(sm + b * a.x_pitch + 16 * c) = make_uint4(0, 0, 0, 0);
        auto norm_pass = [&](int p, const uint2& wv, float eps, bool res, bool last) {
#pragma unroll
          for (int b = 0; b < kNormTokens; b++) {
            float ss = 0.f;
#pragma unroll
            for (int e = 0; e < 4; e++) ss += v[b][e] * v[b][e];
            ss = warp_sum(ss);
            if (lane == 0) red[(b * 2 + p) * 16 + warp] = ss;
          }
          __syncthreads();
          float w[4];
          four(wv, w);
#pragma unroll
          for (int b = 0; b < kNormTokens; b++) {
            if (b >= a.B) break;
            const float inv = rsqrtf(warp_sum(lane < norm_warps ? red[(b * 2 + p) * 16 + lane] : 0.f) / (float)a.K + eps);
            uint16_t o[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const float n = rbf(v[b][e] * inv * (1.0f + w[e]));
              o[e] = res ? f2bf(r[b][e] + n) : f2bf(n);
              v[b][e] = norm_at < a.K ? bf2f(o[e]) : 0.f;
            }
            if (norm_at >= a.K) continue;
            const uint2 bits = make_uint2(o[0] | (uint32_t)o[1] << 16, o[2] | (uint32_t)o[3] << 16);
            if (last) *reinterpret_cast<uint2*>(sm + b * a.x_pitch + 2 * norm_at) = bits;
            else if (blockIdx.x == 0) *reinterpret_cast<uint2*>(a.norm_out + (size_t)b * a.K + norm_at) = bits;
          }
        };
        norm_pass(0, norm_wv, a.norm_eps, a.norm_res != nullptr, !a.norm_w2);
        if (a.norm_w2) norm_pass(1, norm_wv2, a.norm_eps2, false, true);
      }
    }
    if (!staged) {
      const int vec = (kb1 - kb0) * 8;  // 16-byte pieces per token
      for (int b = warp; b < kTok; b += warps) {
        const uint16_t* src = a.x + (b < a.B ? (size_t)b * a.K : 0) + kb0 * kBlk;
        const uint32_t dst = x_addr + (uint32_t)(b * a.x_pitch);
#pragma unroll 4
        for (int c = lane; c < vec; c += 32) cp_async16(dst + 16 * c, src + 8 * c, b < a.B);
      }
      cp_commit();
    }
    cp_wait<0>();
  }
  if (MODE == kRope && pos_now != pos_seen) rope_angle(pos_now);
  if (MODE != kStream && (int)threadIdx.x < a.rt * kTileRows) scale_s[threadIdx.x] = bf2f(scale_r);
  __syncthreads();

  int stage = 0, kb = 0, tile = tile0;
  // Sums of this warp: [16-row half][tile of eight columns][...]. Of slices (ci): columns are the slices of two tokens, 2 t + tig / 2 for this
  // lane; else (cs) eight tokens.
  // Independent chains of accumulation where the tokens leave room: a dependent matrix instruction waits 28 cycles.
  constexpr int kTiles = kTok / 8, kSets = kTiles > 2 ? 1 : kTiles == 2 ? 2 : 4;
  float cs[kSets][2][kTiles][4];
  int ci[2][NT][4];
  auto& c = cs[0];
  float best_v[kTiles][2], best_sliced_v[NT];
  int best_i[kTiles][2], best_sliced_i[NT];
#pragma unroll
  for (int t = 0; t < kTiles; t++) {
    best_v[t][0] = best_v[t][1] = -INFINITY;
    best_i[t][0] = best_i[t][1] = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int q = 0; q < kSets; q++) cs[q][0][t][j] = cs[q][1][t][j] = 0.f;
  }
#pragma unroll
  for (int t = 0; t < NT; t++) {
    best_sliced_v[t] = -INFINITY;
    best_sliced_i[t] = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < 4; j++) ci[0][t][j] = ci[1][t][j] = 0;
  }
  // Every token takes one of the two forms by what is in its own row, so its result does not depend on the tokens beside it.
  uint32_t sliced_tokens = 0;  // a bit each
  int shift[NT] = {};          // of this lane's token in each tile
  if constexpr (SLICED) {
    for (int b = 0; b < a.B; b++) sliced_tokens |= (uint32_t)(shifts[b] != kNoSlices) << b;
#pragma unroll
    for (int t = 0; t < NT; t++) shift[t] = sliced_tokens >> (2 * t + (tig >> 1)) & 1 ? shifts[2 * t + (tig >> 1)] : 0;
  }
  // a lane's finished sum of row 16 mt + 8 (tig % 2) + g for its token of tile t (two lanes hold two slices each and finish a row each)
  auto finished = [&](int mt, int t) {
    const float lo = (float)ci[mt][t][0] + 256.f * (float)ci[mt][t][1], hi = (float)ci[mt][t][2] + 256.f * (float)ci[mt][t][3];  // rows g, g + 8
    const float other = __shfl_xor_sync(0xffffffffu, tig & 1 ? lo : hi, 1);
    const float v = tig & 1 ? 65536.f * hi + other : 65536.f * other + lo;
    const int first = min(shift[t], 126);
    return v * pow2(-first) * pow2(first - shift[t]);
  };
  auto fold = [&]() {  // the chains into the first, which the others start from zero after
    if (kSets == 1) return;
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
      for (int t = 0; t < kTiles; t++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (kSets == 4) c[mt][t][j] = (c[mt][t][j] + cs[1 % kSets][mt][t][j]) + (cs[2 % kSets][mt][t][j] + cs[3 % kSets][mt][t][j]);
          else c[mt][t][j] += cs[1 % kSets][mt][t][j];
#pragma unroll
          for (int q = 1; q < kSets; q++) cs[q][mt][t][j] = 0.f;
        }
  };
  // xrow: this lane's first staged activations. (Positions and addresses outside: with them in here the compiler made the forms of 25 to 32
  // tokens 2 % slower.)
  auto multiply = [&](auto of_slices, uint32_t xrow, int x_pitch) {
    constexpr bool kInts = decltype(of_slices)::value;
    for (int i = 0; i < total; i++) {
      if (MODE == kStream) {  // the ring is a.stages deep and one group is committed per block from here on
        if (kInts || i >= a.stages) cp_wait<kStreamStages - 1>();
        __syncwarp();
      }
      const uint32_t src = ring + stage * kStageBytes + g * kBlk + tig * 16;
      const uint4 w0 = lds128(src), w1 = lds128(src + 8 * kBlk), w2 = lds128(src + 16 * kBlk), w3 = lds128(src + 24 * kBlk);
      if (MODE == kStream) {
        __syncwarp();  // read by every lane before any of them refills the stage
        if (issued < total) {
          issue();
          issued++;
        }
        cp_commit();
      }
      if constexpr (kInts) {
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const uint4 x = lds128(xrow + (uint32_t)(t * 8 * x_pitch + kb * kBlk));
          mma_s8(ci[0][t], w0.x, w1.x, w0.y, w1.y, x.x, x.y);
          mma_s8(ci[1][t], w2.x, w3.x, w2.y, w3.y, x.x, x.y);
          mma_s8(ci[0][t], w0.z, w1.z, w0.w, w1.w, x.z, x.w);
          mma_s8(ci[1][t], w2.z, w3.z, w2.w, w3.w, x.z, x.w);
        }
      } else {
        const uint32_t ww[4][4] = {{w0.x, w0.y, w0.z, w0.w}, {w1.x, w1.y, w1.z, w1.w}, {w2.x, w2.y, w2.z, w2.w}, {w3.x, w3.y, w3.z, w3.w}};
        uint4 x0[kTiles], x1[kTiles];
#pragma unroll
        for (int t = 0; t < kTiles; t++) {
          const uint32_t xa = xrow + (uint32_t)(t * 8 * x_pitch + kb * kBlk * 2);
          x0[t] = lds128(xa);
          x1[t] = lds128(xa + 16);
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
          uint32_t f[4][2];
#pragma unroll
          for (int r = 0; r < 4; r++) s8x4_to_bf16x4(ww[r][m], f[r][0], f[r][1]);
#pragma unroll
          for (int t = 0; t < kTiles; t++) {
            const uint32_t b0 = m == 0 ? x0[t].x : m == 1 ? x0[t].z : m == 2 ? x1[t].x : x1[t].z;
            const uint32_t b1 = m == 0 ? x0[t].y : m == 1 ? x0[t].w : m == 2 ? x1[t].y : x1[t].w;
            mma_bf16(cs[m % kSets][0][t], f[0][0], f[1][0], f[0][1], f[1][1], b0, b1);
            mma_bf16(cs[m % kSets][1][t], f[2][0], f[3][0], f[2][1], f[3][1], b0, b1);
          }
        }
      }
      if (++stage == a.stages) stage = 0;
      if (++kb == nb) {
        kb = 0;
        if (!kInts) fold();
        if (MODE == kStream) {
          auto take = [&](int n, float s, float sum, int b, float& best, int& at) {
            const float v = sum * s;
            if (n >= a.N || b >= a.B || (SLICED && (sliced_tokens >> b & 1) != kInts)) return;
            if (a.y_f32) ((float*)a.y)[(size_t)b * a.N + n] = v;
            else ((uint16_t*)a.y)[(size_t)b * a.N + n] = f2bf(v);
            if (v > best) {  // a warp's rows come in rising order: ties keep the lower index
              best = v;
              at = n;
            }
          };
          if constexpr (kInts) {
#pragma unroll
            for (int mt = 0; mt < 2; mt++) {
              const int n = tile * kTileRows + 16 * mt + 8 * (tig & 1) + g;
              const float s = n < a.N ? bf2f(__ldg(a.scale + n)) : 0.f;
#pragma unroll
              for (int t = 0; t < NT; t++) {
                take(n, s, finished(mt, t), 2 * t + (tig >> 1), best_sliced_v[t], best_sliced_i[t]);
#pragma unroll
                for (int j = 0; j < 4; j++) ci[mt][t][j] = 0;
              }
            }
          } else {
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const int n = tile * kTileRows + 16 * mt + 8 * h + g;
                const float s = n < a.N ? bf2f(__ldg(a.scale + n)) : 0.f;
#pragma unroll
                for (int t = 0; t < kTiles; t++)
#pragma unroll
                  for (int e = 0; e < 2; e++) {
                    take(n, s, c[mt][t][2 * h + e], 8 * t + 2 * tig + e, best_v[t][e], best_i[t][e]);
                    c[mt][t][2 * h + e] = 0.f;
                  }
              }
          }
          tile += tile_step;
        }
      }
    }
  };
  if constexpr (SLICED) {
    if (sliced_tokens) multiply(std::true_type(), x_addr + (uint32_t)(g * a.x_pitch + tig * 16), a.x_pitch);
    if (sliced_tokens != (1u << a.B) - 1) {  // once more for the rows left to bf16, staged where the slices were (they take half of that)
      __syncthreads();
      const int pitch = (a.K * 2 + 127) / 128 * 128 + 16;
      for (int b = warp; b < a.B; b += warps)
        for (int v = lane; v < a.K / 8; v += 32) cp_async16(x_addr + (uint32_t)(b * pitch + 16 * v), a.x + (size_t)b * a.K + 8 * v, true);
      cp_commit();
      if (sliced_tokens) {
        is_tile = tile0;
        is_kb = is_stage = 0;
        for (issued = 0; issued < a.stages && issued < total; issued++) {
          issue();
          cp_commit();
        }
      }
      cp_wait<0>();
      __syncthreads();
      stage = kb = 0;
      tile = tile0;
      multiply(std::false_type(), x_addr + (uint32_t)(min(g, a.B - 1) * pitch + tig * 32), pitch);
    }
  } else {
    multiply(std::false_type(), x_addr + (uint32_t)(g * a.x_pitch + (wb0 - kb0) * kBlk * 2 + tig * 32), a.x_pitch);
  }

  if constexpr (MODE == kStream) {
    if (!a.cand_v) return;
    // best of the block per token, lowest row on ties
    __syncthreads();
    float* sv = reinterpret_cast<float*>(sm);
    int* si = reinterpret_cast<int*>(sm) + 16 * kTok;
    // a lane's best of a token, against those of the other lanes that hold the token
    auto leave = [&](float v, int n, int b, bool sliced) {
#pragma unroll
      for (int o = sliced ? 1 : 4; o < 32; o = o == 1 ? 4 : o << 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int on = __shfl_xor_sync(0xffffffffu, n, o);
        if (ov > v || (ov == v && on < n)) {
          v = ov;
          n = on;
        }
      }
      if (g == 0 && (!SLICED || (b < a.B && (sliced_tokens >> b & 1) == sliced))) {
        sv[warp * kTok + b] = v;
        si[warp * kTok + b] = n;
      }
    };
    if constexpr (SLICED)
#pragma unroll
      for (int t = 0; t < NT; t++) leave(best_sliced_v[t], best_sliced_i[t], 2 * t + (tig >> 1), true);
#pragma unroll
    for (int t = 0; t < kTiles; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) leave(best_v[t][e], best_i[t][e], 8 * t + 2 * tig + e, false);
    __syncthreads();
    if ((int)threadIdx.x < a.B) {
      float v = sv[threadIdx.x];
      int n = si[threadIdx.x];
      for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
        const float ov = sv[w * kTok + threadIdx.x];
        const int on = si[w * kTok + threadIdx.x];
        if (ov > v || (ov == v && on < n)) {
          v = ov;
          n = on;
        }
      }
      a.cand_v[threadIdx.x * gridDim.x + blockIdx.x] = v;
      a.cand_i[threadIdx.x * gridDim.x + blockIdx.x] = n;
    }
    return;
  } else {
  // ---- the groups' sums meet: [tile of the block][group of the block][32 rows][tokens], over the staged operands ----
  __syncthreads();
  float* sums = reinterpret_cast<float*>(sm);
  float* mine = sums + (rt * a.kg + kg) * (kTileRows * kPitch);
#pragma unroll
  for (int mt = 0; mt < 2; mt++)
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int j = 0; j < 4; j++) mine[(16 * mt + g + 8 * (j >> 1)) * kPitch + 8 * t + 2 * tig + (j & 1)] = c[mt][t][j];
  __syncthreads();
  // the block's groups, in order
  auto block_sum = [&](int r_t, int row, int tok) {
    const float* at = sums + r_t * a.kg * (kTileRows * kPitch) + row * kPitch + tok;
    float v = at[0];
#pragma unroll 4
    for (int k = 1; k < a.kg; k++) v += at[k * (kTileRows * kPitch)];
    return v;
  };
  auto tile_of = [&](int i) { return (i * a.inv_b) >> 16; };  // i / B for i < 16 * 32
  // Results are numbered i = tile of the block * B + token, 32 rows each. In a cluster block i % ck finishes result i: the others
  // store their sums into its shared memory, 128 contiguous bytes a warp (reading them over one by one, a word per lane
  // and request, took up to 40 us), and it adds the blocks' sums in order.
  float* recv = reinterpret_cast<float*>(sm + a.recv_off);  // [block of the cluster][i / ck][32]
  const int share = (a.rt * a.B + a.ck - 1) >> ck_log2;
  if (MODE != kRope && a.ck > 1) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    for (int i = warp; i < a.rt * a.B; i += warps)
      st_peer(smem_u32(recv + (rank * share + (i >> ck_log2)) * 32 + lane), i & (a.ck - 1), block_sum(tile_of(i), lane, i - tile_of(i) * a.B));
    cluster_sync();
  }
  auto sum_of = [&](int i, int row) {
    if (a.ck <= 1) return block_sum(tile_of(i), row, i - tile_of(i) * a.B);
    float v = recv[(i >> ck_log2) * 32 + row];
    for (int q = 1; q < a.ck; q++) v += recv[(q * share + (i >> ck_log2)) * 32 + row];
    return v;
  };
  if constexpr (MODE == kStore) {
    for (int i = warp * a.ck + rank; i < a.rt * a.B; i += warps * a.ck) {
      const int r_t = tile_of(i), b = i - r_t * a.B, n = (row_block * a.rt + r_t) * kTileRows + lane;
      const float v = sum_of(i, lane) * scale_s[r_t * kTileRows + lane];
      if (n >= a.N) continue;
      if (a.y_f32) ((float*)a.y)[(size_t)b * a.N + n] = v;
      else ((uint16_t*)a.y)[(size_t)b * a.N + n] = f2bf(v);
    }
  } else if constexpr (MODE == kGeglu) {
    const int I = a.N / 2, r = lane & 15;  // half a warp per token
    const int step = 2 * warps * a.ck, count = a.rt * a.B;
    auto finish = [&](int i0, auto in_flight) {
      constexpr int U = decltype(in_flight)::value;
      float gate[U], up[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + u * step < count ? i0 + u * step : i0;
        const float* sc = scale_s + tile_of(i) * kTileRows;
        gate[u] = rbf(sum_of(i, r) * sc[r]);
        up[u] = rbf(sum_of(i, 16 + r) * sc[16 + r]);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + u * step, r_t = tile_of(i), n = (row_block * a.rt + r_t) * 16 + r;
        if (i < count && n < I) ((uint16_t*)a.y)[(size_t)(i - r_t * a.B) * I + n] = f2bf(rbf(gelu_tanh(gate[u])) * up[u]);
      }
    };
    int i0 = (warp * 2 + (lane >> 4)) * a.ck + rank;
    for (; i0 + step < count; i0 += 2 * step) finish(i0, std::integral_constant<int, 2>());
    if (i0 < count) finish(i0, std::integral_constant<int, 1>());
  } else {
    // one head of 256 rows per cluster, 32 rows per block: lane = row
    // rank = 32 rows of the head; rows i and i + 128 rotate together, so blocks part and part ^ 4 exchange their values
    float* ss = recv;            // [block][tokens] sums of squares
    float* nv = ss + 8 * kTok;   // [tokens][32] the partner's values
    const float scale = scale_s[lane];
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    float own[kRopeTokens];
#pragma unroll
    for (int u = 0; u < kRopeTokens; u++) {
      const int b = warp + u * warps;
      if (b >= a.B) break;
      own[u] = rbf(block_sum(0, lane, b) * scale);
      st_peer(smem_u32(nv + b * 32 + lane), part ^ 4, own[u]);
      const float q = warp_sum(own[u] * own[u]);
      if (lane < 8) st_peer(smem_u32(ss + part * kTok + b), lane, q);
    }
    cluster_sync();
#pragma unroll
    for (int u = 0; u < kRopeTokens; u++) {
      const int b = warp + u * warps;
      if (b >= a.B) break;
      float v = own[u];
      if (is_q || is_k) {
        float q = 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) q += ss[k * kTok + b];
        const float inv = rsqrtf(q / 256.0f + a.eps);
        const float mine = rbf(own[u] * inv * (1.0f + bf2f(norm_w))), other = rbf(nv[b * 32 + lane] * inv * (1.0f + bf2f(norm_w_other)));
        v = part < 4 ? mine * rope_c - other * rope_s : mine * rope_c + other * rope_s;
      }
      uint16_t* dst = is_q ? a.q_out + ((size_t)b * a.n_q + head) * 256 : (is_k ? a.kcache : a.vcache) + ((size_t)b * a.T + pos) * 256;
      dst[part * 32 + lane] = f2bf(v);
    }
  }
  }
}

// Head norm, RoPE and cache append on finished q/k/v values, head size 256: a warp per (sequence, head). The same arithmetic in the
// same order as the epilogue of linear_w8_kernel.
__global__ void __launch_bounds__(128) rope_head_kernel(const uint16_t* __restrict__ qkv, const int32_t* __restrict__ pos_p,
                                                        const uint16_t* __restrict__ qw, const uint16_t* __restrict__ kw,
                                                        uint16_t* __restrict__ q_out, uint16_t* __restrict__ kcache,
                                                        uint16_t* __restrict__ vcache, int B, int n_q, int n_kv, int T, float theta, float eps) {
  const int heads = n_q + 2 * n_kv, lane = threadIdx.x & 31;
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= B * heads) {
    grid_dependency_wait();
    return;
  }
  const int b = item / heads, h = item - b * heads;
  const bool is_q = h < n_q, is_k = !is_q && h < n_q + n_kv;
  float w[8];
#pragma unroll
  for (int j = 0; j < 8; j++) w[j] = (is_q || is_k) ? 1.0f + bf2f(__ldg((is_q ? qw : kw) + 32 * j + lane)) : 0.f;
  grid_dependency_wait();
  grid_dependency_release();
  int pos = __ldcg(pos_p);
  pos = pos < 0 ? 0 : (pos >= T ? T - 1 : pos);
  float v[8], s = 0.f;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    v[j] = bf2f(__ldcg(qkv + (size_t)item * 256 + 32 * j + lane));
    s += warp_sum(v[j] * v[j]);
  }
  uint16_t* dst = is_q ? q_out + ((size_t)b * n_q + h) * 256
                       : (is_k ? kcache : vcache) + (((size_t)b * T + pos) * n_kv + (is_k ? h - n_q : h - n_q - n_kv)) * 256;
  if (!is_q && !is_k) {
#pragma unroll
    for (int j = 0; j < 8; j++) dst[32 * j + lane] = f2bf(v[j]);
    return;
  }
  const float inv = rsqrtf(s / 256.0f + eps);
#pragma unroll
  for (int j = 0; j < 8; j++) v[j] = rbf(v[j] * inv * w[j]);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float inv_freq = powf(theta, -(float)(32 * j + lane) / 128.0f);
    float sn, cs;
    sincosf((float)pos * inv_freq, &sn, &cs);
    dst[32 * j + lane] = f2bf(v[j] * cs - v[j + 4] * sn);
    dst[128 + 32 * j + lane] = f2bf(v[j + 4] * cs + v[j] * sn);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// One query per head against the cache of its sequence (one KV head of 256, up to 4 query heads). A cluster of eight blocks is
// one sequence; a block takes an eighth of the visible keys, a warp 16 keys at a time, copied to shared memory at once (rows
// 64 and 16 bytes apart modulo 128: no bank is hit twice): scores = heads (4 of 16 rows used) x 8 keys, whose accumulator layout is at once the operand layout of the
// second product, values (16 dims) x heads. The probabilities enter that product as three bf16 terms whose sum is the fp32
// number exactly (columns 0-3 and 4-7 of one instruction, columns 0-3 of another), so nothing is lost against an fp32
// product. Warps merge in shared memory, blocks through distributed shared memory: one launch, no partial sums in memory.
// What bounds it is the cache's way from HBM: its lines are prefetched before the wait for the kernel ahead.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kAttnBlocks = 8, kAttnWarps = 4, kAttnCol = 256 + 8;
constexpr int kKeyPitch = 512 + 64, kValPitch = 512 + 16, kAttnWarpBytes = 16 * (kKeyPitch + kValPitch);
static_assert(8 * kAttnCol * 4 <= kAttnWarpBytes, "the warps' results take the place of their keys and values");

__global__ void __launch_bounds__(kAttnWarps * 32, 3) attn_cluster_kernel(const uint16_t* __restrict__ q, const int32_t* __restrict__ pos_p,
                                                                          const uint16_t* kcache, const uint16_t* vcache,
                                                                          uint16_t* __restrict__ out, int n_q, int T, int window, float scale, int early) {
  extern __shared__ __align__(128) unsigned char kv_s[];  // [warp][16 keys, 16 values], later [warp][8 columns][kAttnCol] results
  __shared__ float part_ml[kAttnWarps][4][2];
  __shared__ float recv_acc[kAttnBlocks][kAttnWarps * 32];  // every block's sums of the outputs this block finishes
  __shared__ float recv_ml[kAttnBlocks][4][2];              // and every block's (max, sum) per head
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first remote store
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int rank = blockIdx.x, b = blockIdx.y;
  int t0, t1, pos;
  auto slice = [&](int p) {
    pos = p < 0 ? 0 : (p >= T ? T - 1 : p);
    const int t_lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int per = ((pos + 1 - t_lo + kAttnBlocks - 1) / kAttnBlocks + 15) & ~15;
    t0 = t_lo + rank * per;
    t1 = min(pos + 1, t0 + per);
  };
  const uint16_t* kc = kcache + (size_t)b * T * 256;
  const uint16_t* vc = vcache + (size_t)b * T * 256;
  const uint32_t ks = smem_u32(kv_s) + warp * kAttnWarpBytes, vs = ks + 16 * kKeyPitch;
  auto copy_row = [&](const uint16_t* src, int t, uint32_t dst) {  // a row is 32 pieces of 16 bytes: one per lane
    cp_async16(dst + lane * 16, src + (size_t)t * 256 + lane * 8, true);
  };
  auto copy = [&](const uint16_t* src, int t, uint32_t dst, int pitch) {
#pragma unroll
    for (int r = 0; r < 16; r++) copy_row(src, min(t + r, t1 - 1), dst + r * pitch);
    cp_commit();
  };
  // The rows of earlier steps are final, so they may be read before the wait when the launch ahead is the append of row pos
  // (early); anything else only pulls them towards L2. What depends on the launch ahead is read again behind the wait.
  slice(__ldcg(pos_p));
  const int pos_seen = pos;
  if (early) {
    if (t0 + 16 * warp < t1) {
      copy(kc, t0 + 16 * warp, ks, kKeyPitch);
      copy(vc, t0 + 16 * warp, vs, kValPitch);
    }
  }
  for (int row = t0 + 16 * (warp + (early ? kAttnWarps : 0)) + (lane & 15); row < t1; row += 16 * kAttnWarps) {
    const uint16_t* p = (lane < 16 ? kc : vc) + (size_t)row * 256;
#pragma unroll
    for (int j = 0; j < 4; j++) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 64 * j));
  }
  grid_dependency_wait();
  grid_dependency_release();
  slice(__ldcg(pos_p));
  const int t_first = t0 + 16 * warp;
  if (!early || pos != pos_seen) {
    cp_wait<0>();
    __syncwarp();
    if (t_first < t1) {
      copy(kc, t_first, ks, kKeyPitch);
      copy(vc, t_first, vs, kValPitch);
    }
  } else if (t_first < t1 && t_first + 16 >= t1 && t1 - 1 == pos) {  // the new row, and its copies that fill the round
    cp_wait<0>();
    __syncwarp();
    for (int r = pos - t_first; r < 16; r++) copy_row(kc, pos, ks + r * kKeyPitch);
    cp_commit();
    for (int r = pos - t_first; r < 16; r++) copy_row(vc, pos, vs + r * kValPitch);
    cp_commit();
  }
  uint4 qf[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    qf[j] = make_uint4(0, 0, 0, 0);
    if (g < n_q) qf[j] = __ldcg(reinterpret_cast<const uint4*>(q + ((size_t)b * n_q + g) * 256 + 32 * j + 8 * t4));
  }
  float m = -INFINITY, l = 0.f, acc[16][4];
#pragma unroll
  for (int j = 0; j < 16; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[j][e] = 0.f;
  for (int t = t_first; t < t1; t += 16 * kAttnWarps) {
    if (t != t_first) {
      __syncwarp();  // every lane has read the round before
      copy(kc, t, ks, kKeyPitch);
      copy(vc, t, vs, kValPitch);
    }
    cp_wait<1>();
    __syncwarp();
    // ---- scores of 2 x 8 keys ----
    float s[2][4];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      uint4 kf[8];
#pragma unroll
      for (int j = 0; j < 8; j++) kf[j] = lds128(ks + (8 * u + g) * kKeyPitch + 64 * j + 16 * t4);
      float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 8; j++) {
        mma_bf16(c0, qf[j].x, 0u, qf[j].y, 0u, kf[j].x, kf[j].y);
        mma_bf16(c1, qf[j].z, 0u, qf[j].w, 0u, kf[j].z, kf[j].w);
      }
#pragma unroll
      for (int e = 0; e < 2; e++) s[u][e] = t + 8 * u + 2 * t4 + e < t1 ? (c0[e] + c1[e]) * scale : -INFINITY;
    }
    float mx = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m, mx), corr = expf(m - m_new);
    m = m_new;
    float p[2][2];
    l *= corr;
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        p[u][e] = expf(s[u][e] - m_new);
        l += p[u][e];
      }
    const float corr0 = __shfl_sync(0xffffffffu, corr, ((2 * t4) & 3) * 4), corr1 = __shfl_sync(0xffffffffu, corr, ((2 * t4 + 1) & 3) * 4);
    uint32_t b_hm[2], b_lo[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      uint16_t hm[2], lo[2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const float x = __shfl_sync(0xffffffffu, p[u][e], lane & 15);
        const float hi = rbf(x), mid = rbf(x - hi);
        hm[e] = g < 4 ? f2bf(hi) : f2bf(mid);
        lo[e] = g < 4 ? f2bf((x - hi) - mid) : (uint16_t)0;
      }
      b_hm[u] = hm[0] | (uint32_t)hm[1] << 16;
      b_lo[u] = lo[0] | (uint32_t)lo[1] << 16;
    }
    // ---- values ----
    cp_wait<0>();
    __syncwarp();
#pragma unroll
    for (int d = 0; d < 4; d++) {
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; k++)
        v[k] = lds128(vs + (2 * t4 + (k & 1) + 8 * (k >> 1)) * kValPitch + 128 * d + 16 * g);
      const uint32_t r[4][4] = {{v[0].x, v[0].y, v[0].z, v[0].w}, {v[1].x, v[1].y, v[1].z, v[1].w}, {v[2].x, v[2].y, v[2].z, v[2].w}, {v[3].x, v[3].y, v[3].z, v[3].w}};
#pragma unroll
      for (int j = 0; j < 4; j++) {  // row g: dim 64 d + 8 g + j, row g + 8: dim 64 d + 8 g + 4 + j
        const uint32_t sel = j & 1 ? 0x7632 : 0x5410;
        const uint32_t a0 = __byte_perm(r[0][j >> 1], r[1][j >> 1], sel), a1 = __byte_perm(r[0][2 + (j >> 1)], r[1][2 + (j >> 1)], sel);
        const uint32_t a2 = __byte_perm(r[2][j >> 1], r[3][j >> 1], sel), a3 = __byte_perm(r[2][2 + (j >> 1)], r[3][2 + (j >> 1)], sel);
        float(&c)[4] = acc[4 * d + j];
        c[0] *= corr0; c[1] *= corr1; c[2] *= corr0; c[3] *= corr1;
        mma_bf16(c, a0, a1, a2, a3, b_hm[0], b_hm[1]);
        mma_bf16(c, a0, a1, a2, a3, b_lo[0], b_lo[1]);
      }
    }
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (t4 == 0 && g < 4) {
    part_ml[warp][g][0] = m;
    part_ml[warp][g][1] = l;
  }
  __syncwarp();
  float(*part)[kAttnCol] = reinterpret_cast<float(*)[kAttnCol]>(kv_s + warp * kAttnWarpBytes);
#pragma unroll
  for (int j = 0; j < 16; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) part[2 * t4 + (e & 1)][16 * j + g + 8 * (e >> 1)] = acc[j][e];
  __syncthreads();
  // warp = head: the block's sums go to the blocks that finish them, 128 contiguous bytes a store
  const int share = n_q * (256 / kAttnBlocks);
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (warp < n_q) {
    float mm = -INFINITY, ll = 0.f, e[kAttnWarps];
#pragma unroll
    for (int w = 0; w < kAttnWarps; w++) mm = fmaxf(mm, part_ml[w][warp][0]);
#pragma unroll
    for (int w = 0; w < kAttnWarps; w++) {
      e[w] = part_ml[w][warp][1] > 0.f ? expf(part_ml[w][warp][0] - mm) : 0.f;
      ll += part_ml[w][warp][1] * e[w];
    }
    if (lane < kAttnBlocks) {
      st_peer(smem_u32(&recv_ml[rank][warp][0]), lane, mm);
      st_peer(smem_u32(&recv_ml[rank][warp][1]), lane, ll);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int i = 32 * k + lane, at = warp * 256 + 32 * k;
      float o = 0.f;
#pragma unroll
      for (int w = 0; w < kAttnWarps; w++) {
        const float* p = reinterpret_cast<const float*>(kv_s + w * kAttnWarpBytes);
        o += (p[warp * kAttnCol + i] + p[(warp + 4) * kAttnCol + i]) * e[w];
      }
      st_peer(smem_u32(&recv_acc[rank][at % share + lane]), at / share, o);
    }
  }
  cluster_sync();
  if ((int)threadIdx.x < share) {
    const int h = (rank * share + threadIdx.x) >> 8, at = (rank * share + threadIdx.x) & 255;
    float mm = -INFINITY;
#pragma unroll
    for (int r = 0; r < kAttnBlocks; r++) mm = fmaxf(mm, recv_ml[r][h][0]);
    float ll = 0.f, o = 0.f;
#pragma unroll
    for (int r = 0; r < kAttnBlocks; r++)
      if (recv_ml[r][h][1] > 0.f) {
        const float e = expf(recv_ml[r][h][0] - mm);
        ll += recv_ml[r][h][1] * e;
        o += recv_acc[r][threadIdx.x] * e;
      }
    // place `at` of a column: tile (d, j) x row
    const int dim = 64 * (at >> 6) + 8 * (at & 7) + 4 * (at >> 3 & 1) + (at >> 4 & 3);
    out[((size_t)b * n_q + h) * 256 + dim] = f2bf(o / ll);
  }
}

// best of the blocks' candidates, [B][count] values and rows: a warp per token
__global__ void __launch_bounds__(32) argmax_candidates_kernel(const float* __restrict__ pv, const int32_t* __restrict__ pi, int count,
                                                               int32_t* __restrict__ out) {
  grid_dependency_wait();
  grid_dependency_release();
  const int b = blockIdx.x;
  float v = -INFINITY;
  int n = 0x7fffffff;
  auto take = [&](float ov, int on) {
    if (ov > v || (ov == v && on < n)) {
      v = ov;
      n = on;
    }
  };
  for (int c = threadIdx.x; c < count; c += 32) take(__ldcg(pv + b * count + c), __ldcg(pi + b * count + c));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) take(__shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, n, o));
  if (threadIdx.x == 0) out[b] = n;
}

// y = [res +] bf16(x * rsqrt(mean(x^2) + eps) * (1 + w)), optionally followed by the same norm (w2, no residual) of y: a block per row, four
// elements a thread, the row in registers (H a multiple of 4, up to 4096).
template <int V>
__global__ void __launch_bounds__(512) rmsnorm_row_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ res,
                                                          const uint16_t* __restrict__ w, uint16_t* __restrict__ out,
                                                          const uint16_t* __restrict__ w2, uint16_t* __restrict__ out2, int H, float eps,
                                                          float eps2) {
  __shared__ float red[2][16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  auto four = [](const uint2& u, float (&f)[4]) {
    f[0] = __uint_as_float(u.x << 16);
    f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16);
    f[3] = __uint_as_float(u.y & 0xffff0000u);
  };
  uint2 wv[V], wv2[V];
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    wv[k] = wv2[k] = make_uint2(0, 0);
    if (i < H) {
      wv[k] = __ldg(reinterpret_cast<const uint2*>(w + i));
      if (w2) wv2[k] = __ldg(reinterpret_cast<const uint2*>(w2 + i));
    }
  }
  // Lets the product behind it in before its own wait: a norm runs for a microsecond, and a product that came only then asked for its
  // weights and scales 2 us after its activations were there. Before its wait the product reads constants, and the position, which it reads
  // again behind it; and what runs before a norm in a chain (the products, the embedding) releases after its wait, so no chain stacks up.
  // One step of the 1B shape at position 1024: 808 -> 748 us (one sequence), 1215 -> 1167 us (32); products that release first, too: 747 / 1210.
  grid_dependency_release();
  grid_dependency_wait();
  const size_t base = (size_t)blockIdx.x * H;
  float v[V][4], r[V][4], ss = 0.f;
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    uint2 u = make_uint2(0, 0), ur = make_uint2(0, 0);
    if (i < H) {
      u = __ldcg(reinterpret_cast<const uint2*>(x + base + i));
      if (res) ur = __ldcg(reinterpret_cast<const uint2*>(res + base + i));
    }
    four(u, v[k]);
    four(ur, r[k]);
#pragma unroll
    for (int e = 0; e < 4; e++) ss += v[k][e] * v[k][e];
  }
  auto total = [&](float s, int slot) {
    s = warp_sum(s);
    if (lane == 0) red[slot][warp] = s;
    __syncthreads();
    return warp_sum(lane < warps ? red[slot][lane] : 0.f);
  };
  const float inv = rsqrtf(total(ss, 0) / (float)H + eps);
  float ss2 = 0.f;
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    float f[4];
    four(wv[k], f);
    uint16_t o[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float n = rbf(v[k][e] * inv * (1.0f + f[e]));
      o[e] = res ? f2bf(r[k][e] + n) : f2bf(n);
      v[k][e] = bf2f(o[e]);
      ss2 += i < H ? v[k][e] * v[k][e] : 0.f;
    }
    if (i < H) *reinterpret_cast<uint2*>(out + base + i) = make_uint2(o[0] | (uint32_t)o[1] << 16, o[2] | (uint32_t)o[3] << 16);
  }
  if (!w2) return;
  const float inv2 = rsqrtf(total(ss2, 1) / (float)H + eps2);
#pragma unroll
  for (int k = 0; k < V; k++) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    float f[4];
    four(wv2[k], f);
    uint16_t o[4];
#pragma unroll
    for (int e = 0; e < 4; e++) o[e] = f2bf(v[k][e] * inv2 * (1.0f + f[e]));
    if (i < H) *reinterpret_cast<uint2*>(out2 + base + i) = make_uint2(o[0] | (uint32_t)o[1] << 16, o[2] | (uint32_t)o[3] << 16);
  }
}

template <int NT, int MODE, bool SLICED>
cudaError_t launch_linear_as(const LinearArgs& a, const LinearShape& s, int cluster, cudaStream_t stream) {
  auto kernel = linear_w8_kernel<NT, MODE, SLICED>;
  static std::atomic<unsigned long long> attr_done{0};
  if (first_use_on_device(attr_done)) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e != cudaSuccess) return e;
    mark_used_on_device(attr_done);
  }
  // a product that leaves half of the SMs idle has them prefetch
  int grid = s.grid;
  if (MODE != kStream && a.next_bytes && grid * 2 <= current_sm_count()) grid = current_sm_count() / cluster * cluster;
  return launch_dependent_cluster(cluster, kernel, dim3(grid), dim3(s.kg * s.rt * 32), (size_t)s.smem, stream, !a.serial, a);
}
template <int MODE>
cudaError_t launch_linear_mode(const LinearArgs& args, const LinearShape& s, cudaStream_t stream) {
  LinearArgs a = args;
  a.kg = s.kg; a.ck = s.ck; a.rt = s.rt; a.stages = s.stages; a.x_pitch = s.x_pitch; a.x_bytes = s.x_bytes; a.side_off = s.side_off; a.scale_off = s.scale_off; a.recv_off = s.recv_off; a.inv_b = (65536 + a.B - 1) / a.B; a.tiles = s.tiles;
  const int cluster = MODE == kRope ? 8 : s.ck;
  a.work_blocks = s.grid;
  if constexpr (MODE == kStream)
    if (s.sliced) switch (ceil_div(a.B * kSlices, 8)) {
      case 2: return launch_linear_as<2, MODE, true>(a, s, cluster, stream);
      case 3: return launch_linear_as<3, MODE, true>(a, s, cluster, stream);
      case 4: return launch_linear_as<4, MODE, true>(a, s, cluster, stream);
      default: return launch_linear_as<1, MODE, true>(a, s, cluster, stream);
    }
  switch (ceil_div(a.B, 8)) {
    case 1: return launch_linear_as<1, MODE, false>(a, s, cluster, stream);
    case 2: return launch_linear_as<2, MODE, false>(a, s, cluster, stream);
    case 3: return launch_linear_as<3, MODE, false>(a, s, cluster, stream);
    default: return launch_linear_as<4, MODE, false>(a, s, cluster, stream);
  }
}

}  // namespace

bool linear_w8_applies(int B, int N, int K, bool f32) { return linear_shape(B, N, K, kStore, current_sm_count(), f32).ok; }
bool linear_geglu_applies(int B, int N, int K) { return N % 2 == 0 && linear_w8_applies(B, N, K, false) && linear_shape(B, N, K, kGeglu, current_sm_count(), false).ok; }
bool linear_rope_applies(int B, int N, int K, int n_q, int n_kv, int D) {
  return n_kv == 1 && D == 256 && N == (n_q + 2) * 256 && linear_w8_applies(B, N, K, false) && linear_shape(B, N, K, kRope, current_sm_count(), false).ok;
}
bool linear_norm_applies(int B, int N, int K, bool geglu) {
  const LinearShape s = linear_shape(B, N, K, geglu ? kGeglu : kRope, current_sm_count(), false);
  return B <= kNormTokens && s.ok && s.ck == 1 && rmsnorm_row_applies(K) && K <= 4 * 512 && s.kg * s.rt >= ceil_div(K / 4, 32);
}
// whether the arg max over fp32 results can ride along, and the candidates' bytes
size_t linear_argmax_scratch(int B, int N, int K) {
  const LinearShape s = linear_shape(B, N, K, kStore, current_sm_count(), true);
  return s.ok && s.tk == 1 ? (size_t)B * s.grid * 8 : 0;
}

cudaError_t launch_linear(const LinearArgs& a, cudaStream_t stream) {
  const LinearShape s = linear_shape(a.B, a.N, a.K, kStore, current_sm_count(), a.y_f32 != 0);
  if (!s.ok) return cudaErrorInvalidConfiguration;
  return s.tk == 1 ? launch_linear_mode<kStream>(a, s, stream) : launch_linear_mode<kStore>(a, s, stream);
}
cudaError_t launch_linear_geglu(const LinearArgs& a, cudaStream_t stream) {
  const LinearShape s = linear_shape(a.B, a.N, a.K, kGeglu, current_sm_count(), false);
  return s.ok ? launch_linear_mode<kGeglu>(a, s, stream) : cudaErrorInvalidConfiguration;
}
cudaError_t launch_linear_rope(const LinearArgs& a, cudaStream_t stream) {
  const LinearShape s = linear_shape(a.B, a.N, a.K, kRope, current_sm_count(), false);
  return s.ok ? launch_linear_mode<kRope>(a, s, stream) : cudaErrorInvalidConfiguration;
}
cudaError_t launch_linear_argmax(LinearArgs a, void* scratch, int32_t* out, cudaStream_t stream) {
  const LinearShape s = linear_shape(a.B, a.N, a.K, kStore, current_sm_count(), a.y_f32 != 0);
  if (!s.ok || s.tk != 1) return cudaErrorInvalidConfiguration;
  a.cand_v = (float*)scratch;
  a.cand_i = (int32_t*)scratch + (size_t)a.B * s.grid;
  const cudaError_t e = launch_linear_mode<kStream>(a, s, stream);
  if (e != cudaSuccess) return e;
  return launch_dependent(argmax_candidates_kernel, dim3(a.B), dim3(32), 0, stream, a.cand_v, a.cand_i, s.grid, out);
}

void launch_rope_heads(const uint16_t* qkv, const int32_t* pos, const uint16_t* qw, const uint16_t* kw, uint16_t* q_out, uint16_t* kcache,
                       uint16_t* vcache, int B, int n_q, int n_kv, int T, float theta, float eps, cudaStream_t stream) {
  launch_dependent(rope_head_kernel, dim3(ceil_div((long long)B * (n_q + 2 * n_kv), 4)), dim3(128), 0, stream, qkv, pos, qw, kw, q_out, kcache, vcache,
                   B, n_q, n_kv, T, theta, eps);
}

void launch_attn_decode(const uint16_t* q, const int32_t* pos, const uint16_t* kcache, const uint16_t* vcache, uint16_t* out, int B, int n_q,
                        int T, int window, float scale, bool early, cudaStream_t stream) {
  static std::atomic<unsigned long long> attr_done{0};
  if (first_use_on_device(attr_done)) {
    cudaFuncSetAttribute(attn_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnWarps * kAttnWarpBytes);
    mark_used_on_device(attr_done);
  }
  launch_dependent_cluster(kAttnBlocks, attn_cluster_kernel, dim3(kAttnBlocks, B), dim3(kAttnWarps * 32), kAttnWarps * kAttnWarpBytes, stream, true, q, pos, kcache, vcache, out,
                           n_q, T, window, scale, early ? 1 : 0);
}

bool rmsnorm_row_applies(int H) { return H % 4 == 0 && H <= 4096; }
void launch_rmsnorm_row(const uint16_t* x, const uint16_t* res, const uint16_t* w, uint16_t* out, const uint16_t* w2, uint16_t* out2, int rows,
                        int H, float eps, float eps2, cudaStream_t stream) {
  const int threads = std::min(512, ceil_div(ceil_div(H, 4), 32) * 32);
  if (H <= 4 * 512) launch_dependent(rmsnorm_row_kernel<1>, dim3(rows), dim3(threads), 0, stream, x, res, w, out, w2, out2, H, eps, eps2);
  else launch_dependent(rmsnorm_row_kernel<2>, dim3(rows), dim3(threads), 0, stream, x, res, w, out, w2, out2, H, eps, eps2);
}

}  // namespace tb200
