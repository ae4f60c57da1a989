// Small convolutions and products (one image, a few hundred rows): warp-level int8 matrix instructions on fragments that
// go from L2 straight to registers.
//
// What bounds such a call is not arithmetic (a whole MobileNetV2 layer on one image is 1..10 M multiply-adds, well under
// a microsecond on any path) but the chain of latencies between the launch and the last store. The persistent tcgen05
// kernel's chain - tensor-map fetch, TMEM allocation, TMA into shared memory, MMA, commit, TMEM read, staging, TMA store -
// takes 5.8 .. 8.3 us per layer however little there is to do. Here a warp owns a 16 x 32 tile of the result, fetches its
// operands with 16-byte loads (all of them in flight at once), multiplies with mma.sync and stores from registers: one
// memory round trip, no barrier. A long K is split over up to eight warps of a block, whose sums meet in shared memory
// once, so that a layer with few result tiles still has enough loads in flight.
// Measured, one image: 3x3 56x56 x 64 -> 64 7.3 -> 3.0 us, 14x14 x 576 -> 96 6.6 -> 2.3 us, 3x3 20x20 x 128 -> 128
// 7.4 -> 2.7 us, 112x112 x 16 -> 96 6.9 -> 4.0 us.
//
// Fragments. The K order of a product is free as long as both operands agree, so lane (g = lane / 4, t = lane % 4) takes
// the 16 contiguous bytes 16 t .. 16 t + 15 of a 64-byte K step of row g: words 0 / 1 of them are its fragment of the
// first k32 instruction, words 2 / 3 of the second. Likewise the columns: fragment column f of instruction j is channel
// 8 (f / 2) + 2 j + f % 2 of the warp's 32, so that a lane ends with eight consecutive channels of a row and stores eight
// bytes. The weights are laid out in exactly that order by conv_small_pack: a warp's load is 512 contiguous bytes.
#include <string.h>

#include <atomic>

#include "dependent_launch.cuh"
#include "device_memory.cuh"
#include "kernels.h"

namespace tb200 {
namespace {

constexpr int kTileM = 16, kTileN = 32, kStepBytes = 64;
constexpr int kSumPitch = kTileN + 4;  // words per row of a partial tile: rows land on different banks

__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Four consecutive channels of one row: rescale, clamp, table, and the residual add; q[j] are the channels' Q4 records.
__device__ __forceinline__ uint32_t finish4(const ConvSmallArgs& a, const int (&acc)[4], const int4 (&q)[4], int chan, const int8_t* lut,
                                            uint32_t other) {
  int r[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (a.epi == 1) {
      r[j] = scale_q4_sign(acc[j], q[j]);
    } else if (a.epi == 2) {
      r[j] = scale_q4(acc[j], q[j]);
    } else {
      const ChanParams cp = a.chan[chan + j];
      r[j] = scale_cp<false>(acc[j] + cp.bias, cp) + a.out_zp;
    }
    r[j] = max(a.clamp_min, min(a.clamp_max, r[j]));
  }
  uint32_t w = pack4(r[0], r[1], r[2], r[3]);
  if (a.lut) w = pack4(lut[(w & 0xff) ^ 0x80], lut[(w >> 8 & 0xff) ^ 0x80], lut[(w >> 16 & 0xff) ^ 0x80], lut[(w >> 24) ^ 0x80]);
  if (a.res) {  // as binary_linear_kernel, clamped after the fraction is dropped
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int h = mad_wide_hi(sx8(other, j) * 256, a.add_m_other, (long long)(sx8(w, j) * 256) * (long long)a.add_m_self + a.add_k);
      r[j] = max(a.add_clamp_min, min(a.add_clamp_max, h >> a.add_f));
    }
    w = pack4(r[0], r[1], r[2], r[3]);
  }
  return w;
}

// up to 8 bytes of a row at a channel offset; `full` = all of them exist and the address is 8-byte aligned
__device__ __forceinline__ void store_bytes(int8_t* p, uint32_t w, int n) {
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (j < n) p[j] = (int8_t)(w >> (8 * j));
}
__device__ __forceinline__ uint32_t load_bytes(const int8_t* p, int n) {
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (j < n) w |= (uint32_t)(uint8_t)p[j] << (8 * j);
  return w;
}

// MODE: what a row of the product is - kRows: lda bytes of memory; kConv: the taps of an output pixel, IC a multiple of 16;
// kStem: the 27 bytes under a 3 x 3 window of 3 channels, one k32 instruction: lane t = 0 .. 2 holds the first eight of the nine
// bytes of kernel row t (consecutive in memory), lane 3 the three ninth bytes.
// U = K steps whose loads are in flight together; SPLIT: several warps share a tile.
enum { kRows = 0, kConv = 1, kStem = 2 };
// RAGGED: rows or channels that are no multiple of 16 bytes - the 16 bytes of a chunk come from five aligned words and may run on
// into the next pixel's, whose weights here are zero.
template <int MODE, int U, bool SPLIT, bool RAGGED>
__global__ void __launch_bounds__(SPLIT ? 256 : 128, SPLIT ? 2 : 4) conv_small_kernel(const ConvSmallArgs a) {
  extern __shared__ int sums[];  // [tiles of the block][warps of a tile][16][kSumPitch], only with more than one warp per tile
  __shared__ int8_t lut[256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int ks_log2 = SPLIT ? a.ks_log2 : 0, ks_n = 1 << ks_log2;
  const int ks = warp & (ks_n - 1), slot = warp >> ks_log2;
  const int tile = blockIdx.x * ((int)(blockDim.x >> 5) >> ks_log2) + slot;
  const int mt = tile / a.n_tiles, nt = tile - mt * a.n_tiles;
  const bool live = mt < a.m_tiles;
  const int8_t* wp = a.w + ((size_t)(live ? nt : 0) * a.steps * 4) * 512 + lane * 16;
  // the channels this thread finishes: eight of two rows, or (several warps per tile) four of every (8 ks_n)-th row
  const int chan = (live ? nt : 0) * kTileN + (SPLIT ? 4 * (lane & 7) : 8 * t);
  int4 q[SPLIT ? 4 : 8];
  if (a.epi) {
#pragma unroll
    for (int j = 0; j < (SPLIT ? 4 : 8); j++) q[j] = __ldg(a.q4 + chan + j);
  }
  if (a.lut)
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = a.lut[i];

  // the two rows of this lane
  int px[2];
  int ih0[2], iw0[2];
  bool row_ok[2];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int row = mt * kTileM + g + 8 * r;
    row_ok[r] = live && row < a.M;
    if (MODE != kRows) {
      const int pix = row_ok[r] ? row : 0;
      const int n = pix / (a.OH * a.OW), rem = pix - n * (a.OH * a.OW), oh = rem / a.OW, ow = rem - oh * a.OW;
      ih0[r] = oh * a.stride - a.pad_t;
      iw0[r] = ow * a.stride - a.pad_l;
      px[r] = ((n * a.H + ih0[r]) * a.W + iw0[r]) * a.IC;  // may lie outside: only dereferenced inside
    } else {
      px[r] = row * a.lda;
    }
  }
  const uint32_t fill = (uint32_t)(a.input_zp & 0xff) * 0x01010101u;  // a tap outside the frame reads the zero point
  auto load_a = [&](int step, uint4 (&v)[2]) {
    const int c = 4 * step + t;  // 16-byte chunk of the K axis (tap-major)
    const bool in_k = c < a.chunks;
    if (MODE == kStem) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        v[r] = make_uint4(fill, fill, 0, 0);
        if (!row_ok[r]) continue;
        if (t < 3) {
          if ((unsigned)(ih0[r] + t) >= (unsigned)a.H) continue;
          const int off = px[r] + t * a.W * 3;
          if (iw0[r] >= 0 && iw0[r] + 2 < a.W && (off & ~3) + 12 <= a.x_bytes) {
            const uint32_t* p = reinterpret_cast<const uint32_t*>(a.x + (off & ~3));
            const uint32_t w0 = p[0], w1 = p[1], w2 = p[2], sh = (uint32_t)(off & 3) * 8;
            v[r].x = __funnelshift_r(w0, w1, sh);
            v[r].y = __funnelshift_r(w1, w2, sh);
          } else {
            uint32_t b[8];
#pragma unroll
            for (int j = 0; j < 8; j++) b[j] = (unsigned)(iw0[r] + j / 3) < (unsigned)a.W ? (uint32_t)(uint8_t)a.x[off + j] : fill & 0xff;
            v[r].x = b[0] | b[1] << 8 | b[2] << 16 | b[3] << 24;
            v[r].y = b[4] | b[5] << 8 | b[6] << 16 | b[7] << 24;
          }
        } else if ((unsigned)(iw0[r] + 2) < (unsigned)a.W) {
          uint32_t b[3];
#pragma unroll
          for (int kh = 0; kh < 3; kh++) b[kh] = (unsigned)(ih0[r] + kh) < (unsigned)a.H ? (uint32_t)(uint8_t)a.x[px[r] + kh * a.W * 3 + 8] : fill & 0xff;
          v[r].x = b[0] | b[1] << 8 | b[2] << 16;
        }
      }
    } else if (MODE == kConv) {
      const int tap = divide_chunk(c, a.by_icb), icb = c - tap * a.icb;
      const int kh = divide_tap(tap, a.inv_kw), kw = tap - kh * a.KW;
      const int off = (kh * a.W + kw) * a.IC + icb * 16;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        v[r] = make_uint4(fill, fill, fill, fill);
        if (in_k && row_ok[r] && (unsigned)(ih0[r] + kh) < (unsigned)a.H && (unsigned)(iw0[r] + kw) < (unsigned)a.W)
          v[r] = RAGGED ? load16_any(a.x, px[r] + off, a.x_bytes) : *reinterpret_cast<const uint4*>(a.x + (px[r] + off));
      }
    } else {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        v[r] = make_uint4(0, 0, 0, 0);
        if (in_k && row_ok[r]) v[r] = RAGGED ? load16_any(a.x, px[r] + c * 16, a.x_bytes) : *reinterpret_cast<const uint4*>(a.x + (px[r] + c * 16));
      }
    }
  };
  int acc[4][4];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[j][i] = 0;

  bool waited = false;
  for (int s0 = ks; s0 < a.steps; s0 += U * ks_n) {
    uint4 b[U][4], v[U][2];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int s = s0 + u * ks_n;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        b[u][j] = make_uint4(0, 0, 0, 0);
        if (s < a.steps) b[u][j] = __ldg(reinterpret_cast<const uint4*>(wp + ((size_t)s * 4 + j) * 512));
      }
    }
    if (!waited) {  // the weights and constants belong to the program: only the activations wait for the launch before
      grid_dependency_wait();
      grid_dependency_release();
      waited = true;
    }
#pragma unroll
    for (int u = 0; u < U; u++) load_a(s0 + u * ks_n, v[u]);
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        mma_s8(acc[j], v[u][0].x, v[u][1].x, v[u][0].y, v[u][1].y, b[u][j].x, b[u][j].y);
        if (MODE != kStem) mma_s8(acc[j], v[u][0].z, v[u][1].z, v[u][0].w, v[u][1].w, b[u][j].z, b[u][j].w);
      }
  }
  if (!waited) grid_dependency_wait();

  if constexpr (!SPLIT) {
    if (a.lut) __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
      if (!row_ok[r]) continue;
      const long long off = (long long)(mt * kTileM + g + 8 * r) * a.ldc + chan;
      const int left = a.N - chan;
      const bool vec = a.vec && left >= 8;
      uint32_t o[2] = {0, 0};
      if (a.res) {
        if (vec) {
          const uint2 ov = *reinterpret_cast<const uint2*>(a.res + off);
          o[0] = ov.x;
          o[1] = ov.y;
        } else {
          o[0] = load_bytes(a.res + off, left);
          o[1] = load_bytes(a.res + off + 4, left - 4);
        }
      }
      uint32_t w[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int four[4] = {acc[2 * h][2 * r], acc[2 * h][2 * r + 1], acc[2 * h + 1][2 * r], acc[2 * h + 1][2 * r + 1]};
        const int4 qs[4] = {q[4 * h], q[4 * h + 1], q[4 * h + 2], q[4 * h + 3]};
        w[h] = finish4(a, four, qs, chan + 4 * h, lut, o[h]);
      }
      if (vec) {
        *reinterpret_cast<uint2*>(a.out + off) = make_uint2(w[0], w[1]);
      } else {
        store_bytes(a.out + off, w[0], left);
        store_bytes(a.out + off + 4, w[1], left - 4);
      }
    }
    return;
  } else {
  // several warps per tile: every warp leaves its sums, then each takes its share of the rows
  int* mine = sums + (warp * kTileM) * kSumPitch;
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int h = 0; h < 2; h++)
      *reinterpret_cast<int4*>(mine + (g + 8 * r) * kSumPitch + 8 * t + 4 * h) =
          make_int4(acc[2 * h][2 * r], acc[2 * h][2 * r + 1], acc[2 * h + 1][2 * r], acc[2 * h + 1][2 * r + 1]);
  __syncthreads();
  if (!live) return;
  const int* first = sums + ((slot << a.ks_log2) * kTileM) * kSumPitch;
  for (int lr = ks * 4 + (lane >> 3); lr < kTileM; lr += 4 * ks_n) {
    const int row = mt * kTileM + lr;
    if (row >= a.M) break;
    int four[4] = {0, 0, 0, 0};
#pragma unroll 4
    for (int k = 0; k < ks_n; k++) {
      const int4 p = *reinterpret_cast<const int4*>(first + (k * kTileM + lr) * kSumPitch + 4 * (lane & 7));
      four[0] += p.x;
      four[1] += p.y;
      four[2] += p.z;
      four[3] += p.w;
    }
    const long long off = (long long)row * a.ldc + chan;
    const int left = a.N - chan;
    if (left <= 0) break;
    const bool vec = a.vec && left >= 4;
    const uint32_t o = !a.res ? 0u : vec ? *reinterpret_cast<const uint32_t*>(a.res + off) : load_bytes(a.res + off, left);
    const int4 qs[4] = {q[0], q[1], q[2], q[3]};
    const uint32_t w = finish4(a, four, qs, chan, lut, o);
    if (vec) *reinterpret_cast<uint32_t*>(a.out + off) = w;
    else store_bytes(a.out + off, w, left);
  }
  }
}

// ---- products of a few dozen rows ----
// Between the sizes above and those that fill the chip with 128-row tiles a product is bound by how fast its weights arrive:
// FullyConnected 64 x 4096 -> 4096 is 17 MB of weights, 2.6 us of HBM time, and took 17.5 us on 32 tiles of the tcgen05 kernel,
// now 9.9.
// A block takes 64 rows x 128 columns and one of ck slices of K (a cluster), so that every SM streams weights. Chunks of 256
// bytes of K - weights in fragment order, rows at a pitch of 64 bytes modulo 128 - pass through three shared-memory stages by
// cp.async, two of them in flight. A warp is 32 columns x one of the chunk's four steps x all 64 rows: a weight fragment
// then serves four instructions (eight warps with two steps each left the shared-memory reads' latency in the open). The sums are integers: they meet in shared memory, within the block and pushed through
// the cluster, and each block of the cluster finishes its share of the rows.
constexpr int kMidM = 64, kMidN = 128, kMidThreads = 512, kMidStages = 3, kMidSteps = 4;
constexpr int kMidPitch = kMidSteps * kStepBytes + 64;
constexpr int kMidX = kMidM * kMidPitch, kMidW = kMidSteps * 2048 * (kMidN / kTileN), kMidStage = kMidX + kMidW;
constexpr int kMidSumPitch = kMidN + 4;  // words
constexpr int kMidRecv = kMidM * kMidN * 4, kMidSmem = kMidStages * kMidStage + kMidRecv;
constexpr int kMidGroups = kMidThreads / 128;  // warps that share a chunk's steps
static_assert(kMidGroups * kMidM * kMidSumPitch * 4 <= kMidStages * kMidStage, "the sums take the stages' place");

__global__ void __launch_bounds__(kMidThreads, 1) rows_mid_kernel(const ConvSmallArgs a) {
  extern __shared__ __align__(128) unsigned char mid_s[];
  __shared__ int8_t lut[256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ck = 1 << a.ks_log2, rank = blockIdx.x & (ck - 1), nb = blockIdx.x >> a.ks_log2, row0 = blockIdx.y * kMidM;
  const int nt = warp & 3, kg = warp >> 2;
  const int s_begin = a.steps * rank >> a.ks_log2, s_end = a.steps * (rank + 1) >> a.ks_log2;  // steps of 64 bytes of K
  const int chunks = (s_end - s_begin + kMidSteps - 1) / kMidSteps;
  if (ck > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first remote store
  const uint32_t base = smem_u32(mid_s);
  // A thread copies piece threadIdx.x of each of the chunk's four weight tiles and pieces of two rows; pointers and limits are kept
  // (worked out anew for every copy they were 230 of 280 instructions per warp and chunk).
  static_assert(kMidThreads == 512 && kMidSteps == 4 && kMidN == 4 * kTileN && kMidM == 64, "the copies below");
  const int w_step = threadIdx.x >> 7, x_row = threadIdx.x >> 4, x_piece = threadIdx.x & 15;
  const int8_t* wp = a.w + ((size_t)nb * 4 * a.steps + s_begin + w_step) * 2048 + (threadIdx.x & 127) * 16;
  const size_t w_tile = (size_t)a.steps * 2048;
  const int w_tiles = min(4, a.n_tiles - 4 * nb);
  const int8_t* xp = a.x + (long long)(row0 + x_row) * a.lda + s_begin * kStepBytes + x_piece * 16;
  const long long x_next = 32ll * a.lda;
  const bool x_ok0 = row0 + x_row < a.M, x_ok1 = row0 + x_row + 32 < a.M;
  int w_left = s_end - s_begin - w_step;                              // steps from this thread's on
  int x_left = min(a.chunks, s_end * 4) - s_begin * 4 - x_piece;      // pieces from this thread's on
  uint32_t w_dst = base + kMidX + threadIdx.x * 16, x_dst = base + x_row * kMidPitch + x_piece * 16;
  const uint32_t w_end = w_dst + kMidStages * kMidStage, x_end = x_dst + kMidStages * kMidStage;
  auto load_w = [&]() {
#pragma unroll
    for (int i = 0; i < 4; i++) cp_async16(w_dst + i * 8192, w_left > 0 && i < w_tiles ? wp + i * w_tile : a.w, w_left > 0 && i < w_tiles);
    wp += kMidSteps * 2048;
    w_left -= kMidSteps;
    w_dst += kMidStage;
    if (w_dst == w_end) w_dst -= kMidStages * kMidStage;
  };
  auto load_x = [&]() {
    cp_async16(x_dst, x_left > 0 && x_ok0 ? xp : a.x, x_left > 0 && x_ok0);
    cp_async16(x_dst + 32 * kMidPitch, x_left > 0 && x_ok1 ? xp + x_next : a.x, x_left > 0 && x_ok1);
    xp += kMidSteps * kStepBytes;
    x_left -= kMidSteps * 4;
    x_dst += kMidStage;
    if (x_dst == x_end) x_dst -= kMidStages * kMidStage;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_w();
  load_w();
  if (a.lut)
    for (int i = threadIdx.x; i < 256; i += kMidThreads) lut[i] = a.lut[i];
  grid_dependency_wait();
  grid_dependency_release();
  load_x();
  load_x();
  int acc[4][4][4];
#pragma unroll
  for (int m = 0; m < 4; m++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[m][j][i] = 0;
  uint32_t stage = base;
  for (int c = 0; c < chunks; c++) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // chunk c has arrived for everyone, and chunk c - 1 has been read by everyone
    if (c + 2 < chunks) {
      load_w();
      load_x();
    } else {
      asm volatile("cp.async.commit_group;" ::: "memory");  // the wait above counts groups
    }
    const uint32_t xs = stage + g * kMidPitch + t * 16, ws = stage + kMidX + nt * 8192 + lane * 16;
    stage = stage == base + (kMidStages - 1) * kMidStage ? base : stage + kMidStage;
#pragma unroll
    for (int u = 0; u < kMidSteps / kMidGroups; u++) {
      const int s = kMidGroups * u + kg;
      uint4 b[4];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = lds128(ws + s * 2048 + j * 512);
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const uint4 v0 = lds128(xs + (16 * m) * kMidPitch + s * kStepBytes), v1 = lds128(xs + (16 * m + 8) * kMidPitch + s * kStepBytes);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          mma_s8(acc[m][j], v0.x, v1.x, v0.y, v1.y, b[j].x, b[j].y);
          mma_s8(acc[m][j], v0.z, v1.z, v0.w, v1.w, b[j].z, b[j].w);
        }
      }
    }
  }
  // the records of the channels this lane finishes: on their way while the sums meet
  const int chan = nb * kMidN + 4 * lane, left = a.N - chan;
  int4 q[4];
  if (a.epi && left > 0)
#pragma unroll
    for (int j = 0; j < 4; j++) q[j] = __ldg(a.q4 + chan + j);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  int* sums = reinterpret_cast<int*>(mid_s);
#pragma unroll
  for (int m = 0; m < 4; m++)
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        *reinterpret_cast<int4*>(sums + (kg * kMidM + 16 * m + g + 8 * r) * kMidSumPitch + nt * 32 + 8 * t + 4 * h) =
            make_int4(acc[m][2 * h][2 * r], acc[m][2 * h][2 * r + 1], acc[m][2 * h + 1][2 * r], acc[m][2 * h + 1][2 * r + 1]);
  __syncthreads();
  const int share_log2 = 6 - a.ks_log2;  // rows a block of the cluster finishes
  int* recv = reinterpret_cast<int*>(mid_s + kMidStages * kMidStage);  // [block of the cluster][its rows][columns]
  auto block_sum = [&](int row, int col) {
    int4 v = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < kMidGroups; k++) {
      const int4 p = *reinterpret_cast<const int4*>(sums + (k * kMidM + row) * kMidSumPitch + col);
      v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
    }
    return v;
  };
  if (ck > 1) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    for (int row = warp; row < kMidM; row += kMidThreads / 32) {
      if (row0 + row >= a.M) break;
      const int4 v = block_sum(row, 4 * lane);
      const uint32_t local = smem_u32(recv + (((rank << share_log2) + (row & ((1 << share_log2) - 1))) * kMidN) + 4 * lane);
      uint32_t remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(row >> share_log2));
      asm volatile("st.shared::cluster.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(remote), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (left <= 0) return;
  for (int r = warp; r < 1 << share_log2; r += kMidThreads / 32) {
    const int row = (rank << share_log2) + r;
    if (row0 + row >= a.M) break;
    int four[4];
    if (ck > 1) {
      four[0] = four[1] = four[2] = four[3] = 0;
      for (int k = 0; k < ck; k++) {
        const int4 v = *reinterpret_cast<const int4*>(recv + ((k << share_log2) + r) * kMidN + 4 * lane);
        four[0] += v.x; four[1] += v.y; four[2] += v.z; four[3] += v.w;
      }
    } else {
      const int4 v = block_sum(row, 4 * lane);
      four[0] = v.x; four[1] = v.y; four[2] = v.z; four[3] = v.w;
    }
    const uint32_t w = finish4(a, four, q, chan, lut, 0u);
    int8_t* o = a.out + (long long)(row0 + row) * a.ldc + chan;
    if (a.vec && left >= 4) *reinterpret_cast<uint32_t*>(o) = w;
    else store_bytes(o, w, left);
  }
}

int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace

int conv_small_steps(int taps, int IC) { return ceil_div((long long)taps * ceil_div(IC, 16), kStepBytes / 16); }
int conv_small_columns(int OC) { return ceil_div(OC, kTileN) * kTileN; }

// The line to the tcgen05 kernel. A warp's tile costs about (steps + 5) * 0.18 ns of the whole chip beyond the 2 us that
// every launch takes (measured over batches of 2 .. 23 of the layers of both networks), the tcgen05 kernel about 7 us up to
// the same sizes: (tiles, steps, here / there in us) 1600, 6: 5.2 / 7.3; 4800, 1: 7.7 / 8.2; 3200, 5: 9.4 / 9.2;
// 3200, 6: 9.9 / 7.4; 2300, 18: 11.2 / 10.9.
constexpr long long kSmallCost = 29000;

bool conv_small_applies(long long M, int OC, int taps, int IC) {
  if (small_kernels_off() || IC < 1 || taps < 1 || taps > kMaxTaps || (long long)taps * ceil_div(IC, 16) > kMaxChunks) return false;
  const long long tiles = (long long)ceil_div(M, kTileM) * ceil_div(OC, kTileN);
  // unaligned rows take five loads for one: worth it up to half of that (3x3 28x28 x 100 -> 77, cost 12 k, 8.8 us against 12.9
  // padded; FullyConnected 500 x 1001 -> 1003, 21 k, 19.4 us against about 11)
  return tiles * (conv_small_steps(taps, IC) + 5) <= (IC % 16 ? kSmallCost / 2 : kSmallCost) && M * IC < (1ll << 30);
}

void conv_small_pack(const int8_t* w, int OC, int taps, int IC, int8_t* out) {
  const int steps = conv_small_steps(taps, IC), n_tiles = ceil_div(OC, kTileN), icb = ceil_div(IC, 16), chunks = taps * icb;
  const long long K = (long long)taps * IC;
  for (int nt = 0; nt < n_tiles; nt++)
    for (int s = 0; s < steps; s++)
      for (int j = 0; j < 4; j++)
        for (int lane = 0; lane < 32; lane++) {
          const int f = lane >> 2, c = 4 * s + (lane & 3);
          const int oc = nt * kTileN + 8 * (f >> 1) + 2 * j + (f & 1);
          int8_t* o = out + ((((size_t)nt * steps + s) * 4 + j) * 32 + lane) * 16;
          memset(o, 0, 16);
          if (oc >= OC || c >= chunks) continue;
          const int tap = c / icb, ic = (c - tap * icb) * 16;
          memcpy(o, w + (size_t)oc * K + (size_t)tap * IC + ic, (size_t)(IC - ic < 16 ? IC - ic : 16));
        }
}

void conv_small_pack_stem(const int8_t* w, int OC, int8_t* out) {
  for (int i = 0; i < conv_small_columns(OC) * kStepBytes; i++) out[i] = 0;
  for (int nt = 0; nt < ceil_div(OC, kTileN); nt++)
    for (int j = 0; j < 4; j++)
      for (int lane = 0; lane < 32; lane++) {
        const int f = lane >> 2, t = lane & 3, oc = nt * kTileN + 8 * (f >> 1) + 2 * j + (f & 1);
        if (oc >= OC) continue;
        int8_t* o = out + (((size_t)nt * 4 + j) * 32 + lane) * 16;
        for (int i = 0; i < (t < 3 ? 8 : 3); i++) o[i] = w[(size_t)oc * 27 + (t < 3 ? 9 * t + i : 9 * i + 8)];
      }
}

cudaError_t launch_conv_small(const ConvSmallArgs& args, cudaStream_t stream) {
  ConvSmallArgs a = args;
  const int taps = a.KH * a.KW;
  a.m_tiles = ceil_div(a.M, kTileM);
  a.n_tiles = ceil_div(a.N, kTileN);
  a.steps = a.mode == kStem ? 1 : conv_small_steps(taps, a.IC);
  a.icb = a.mode == kStem ? 1 : ceil_div(a.IC, 16);
  a.chunks = taps * a.icb;
  a.by_icb = chunk_divisor(a.icb);
  a.inv_kw = tap_divisor(a.KW);
  a.vec = a.ldc % 8 == 0 && ((uintptr_t)a.out & 7) == 0 && ((uintptr_t)a.res & 7) == 0;
  // K is split over 2 or 4 warps while the grid stays within about twelve warps per SM, over 8 (whose sums take longer to
  // meet) only up to six. One layer, us with 1 / 2 / 4 / 8 warps per tile: 98 tiles, 3 steps 3.0 / 2.3 / 2.0 / 2.1;
  // 392 tiles, 9 steps 4.4 / 3.6 / 3.0 / 4.9; 100 tiles, 18 steps 6.7 / 3.9 / 2.9 / 2.7; 1600 tiles, 3 steps 4.5 / 5.7 / 6.4.
  const long long tiles = (long long)a.m_tiles * a.n_tiles;
  a.ks_log2 = 0;
  while (a.ks_log2 < 3 && (1 << a.ks_log2) < a.steps && (tiles << (a.ks_log2 + 1)) <= (a.ks_log2 == 2 ? 6ll : 12ll) * current_sm_count())
    a.ks_log2++;
  const int ks_n = 1 << a.ks_log2;
  const int per_warp = ceil_div(a.steps, ks_n);
  const int warps = ks_n > 4 ? ks_n : 4;
  const dim3 grid((unsigned)ceil_div(tiles, warps / ks_n)), block(warps * 32);
  const size_t smem = ks_n > 1 ? (size_t)warps * kTileM * kSumPitch * 4 : 0;
  const int u = per_warp < 3 ? per_warp : 3;  // more than three steps in flight do not fit 128 registers
  using Kernel = void (*)(ConvSmallArgs);
  static const Kernel kernels[2][2][2][3] = {  // [ragged][convolution][split][U - 1]
      {{{conv_small_kernel<kRows, 1, false, false>, conv_small_kernel<kRows, 2, false, false>, conv_small_kernel<kRows, 3, false, false>}, {conv_small_kernel<kRows, 1, true, false>, conv_small_kernel<kRows, 2, true, false>, conv_small_kernel<kRows, 3, true, false>}},
       {{conv_small_kernel<kConv, 1, false, false>, conv_small_kernel<kConv, 2, false, false>, conv_small_kernel<kConv, 3, false, false>}, {conv_small_kernel<kConv, 1, true, false>, conv_small_kernel<kConv, 2, true, false>, conv_small_kernel<kConv, 3, true, false>}}},
      {{{conv_small_kernel<kRows, 1, false, true>, conv_small_kernel<kRows, 2, false, true>, conv_small_kernel<kRows, 3, false, true>}, {conv_small_kernel<kRows, 1, true, true>, conv_small_kernel<kRows, 2, true, true>, conv_small_kernel<kRows, 3, true, true>}},
       {{conv_small_kernel<kConv, 1, false, true>, conv_small_kernel<kConv, 2, false, true>, conv_small_kernel<kConv, 3, false, true>}, {conv_small_kernel<kConv, 1, true, true>, conv_small_kernel<kConv, 2, true, true>, conv_small_kernel<kConv, 3, true, true>}}}};
  const bool ragged = a.IC % 16 != 0;
  const Kernel kernel = a.mode == kStem ? conv_small_kernel<kStem, 1, false, false> : kernels[ragged][a.mode == kConv][ks_n > 1][u - 1];
  return launch_dependent(kernel, grid, block, smem, stream, a);
}

namespace {
// log2 of the K slices: while they fill idle SMs and a slice keeps two chunks; clusters of eight are slower even where they
// fit (64 x 4096 -> 4096, us by slices: 20.2 / 13.4 / 9.9 / 19.7)
int mid_slices(long long M, int N, int K) {
  const long long blocks = (long long)ceil_div(N, kMidN) * ceil_div(M, kMidM);
  const int steps = conv_small_steps(1, K);
  int ks = 0;
  while (ks < 2 && blocks << (ks + 1) <= current_sm_count() && steps >> (ks + 1) >= 2 * kMidSteps) ks++;
  return ks;
}
}  // namespace
// A chunk takes about 1.1 us, the tcgen05 kernel about 0.9 us for the same K but a few more to start: ahead of it with K split
// over blocks, or with a short K while every block has an SM of its own. Here / there in us: 64 x 4096 -> 4096 9.9 / 17.5,
// 128 x 4096 -> 4096 13.8 / 17.8, 256 x 1024 -> 4096 9.0 / 10.2, 128 x 2048 -> 8192 13.1 / 14.8; without either
// 256 x 4096 -> 4096 21.3 / 18.4, 128 x 8192 -> 8192 37.7 / 30.8.
bool rows_mid_applies(long long M, int N, int K) {
  if (small_kernels_off() || K % 16 != 0 || M <= 4 || N < 256 || K < 512 || K > (1 << 20)) return false;
  const long long blocks = (long long)ceil_div(N, kMidN) * ceil_div(M, kMidM);
  return blocks <= current_sm_count() && (mid_slices(M, N, K) > 0 || K <= 2560);
}
cudaError_t launch_rows_mid(const ConvSmallArgs& args, cudaStream_t stream) {
  ConvSmallArgs a = args;
  a.n_tiles = ceil_div(a.N, kTileN);
  a.steps = conv_small_steps(1, a.IC);
  a.chunks = a.IC / 16;
  a.vec = a.ldc % 4 == 0 && ((uintptr_t)a.out & 3) == 0;
  const int nb = ceil_div(a.N, kMidN), mb = ceil_div(a.M, kMidM);
  a.ks_log2 = mid_slices(a.M, a.N, a.IC);
  static std::atomic<unsigned long long> attr_done{0};
  if (first_use_on_device(attr_done)) {
    const cudaError_t e = cudaFuncSetAttribute(rows_mid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMidSmem);
    if (e != cudaSuccess) return e;
    mark_used_on_device(attr_done);
  }
  return launch_dependent_cluster(1 << a.ks_log2, rows_mid_kernel, dim3((unsigned)(nb << a.ks_log2), (unsigned)mb), dim3(kMidThreads), (size_t)kMidSmem,
                                  stream, true, a);
}

}  // namespace tb200
