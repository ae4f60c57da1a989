// How a product of decode_linear.cu is cut into warps, blocks and clusters, and what lies where in a block's shared memory.
// Host code only, so that the layout can be checked without a GPU.
//
// Shared memory of a block, in order:
//   [0, x_bytes)                  staged activations: rows, behind them room for the sums of a norm in front; or slices, and a shift per token
//   [x_bytes, + rings)            every warp's weight ring; both are overwritten by the groups' sums once all warps have multiplied
//   [scale_off, + rt * 32 * 4)    scales of the block's rows
//   [recv_off, smem)              what other blocks of the cluster store into this one: nothing else uses it, because a peer that
//                                 is ahead stores while this block is still staging or multiplying
#pragma once
#include <algorithm>

namespace tb200 {

// modes of linear_w8_kernel
enum { kStore = 0, kGeglu = 1, kRope = 2, kStream = 3 };
constexpr int kTileRows = 32, kBlk = 64, kStageBytes = kTileRows * kBlk, kStreamStages = 4;
constexpr int kRopeTokens = 8;  // most tokens a warp finishes in the RoPE epilogue
constexpr int kSmemMax = 227 * 1024 - 1024;
// Up to kSlicedTokens tokens the product over the vocabulary (a stream with fp32 results) multiplies integers: a bf16 activation is four int8 slices of a 31-bit
// fixed-point number, a slice a column of the instruction. Its weights then need no conversion (where the slices leave room for the warps:
// linear_shape). The products of the layers keep bf16: their
// results are rounded to bf16 and go through every layer behind them, where two sums that differ in the last bit of fp32 end almost a
// percent apart.
// Up to kNormTokens the norm in front of a product runs in it.
constexpr int kSlicedTokens = 8, kSlices = 4, kNormTokens = 2;

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// groups of K of a product: enough warps to ask for every weight at once, none without a 64-byte block
inline int linear_groups(int N, int K) {
  const int tiles = ceil_div(N, kTileRows), blocks = K / kBlk;
  const int cap = K <= 4096 ? 16 : 32;
  int tk = 1;
  while (tk * 2 <= blocks && tk < cap && (long long)tiles * tk * 2 <= 12 * 148) tk *= 2;
  return tk;
}

struct LinearShape {
  int tk, kg, ck, rt, stages, x_pitch, x_bytes, side_off, scale_off, recv_off, smem, tiles, grid;
  bool ok, sliced;
};

// bytes other blocks store into one: the RoPE epilogue's sums of squares and partner values, or the sums of a cluster's K slices
inline int linear_recv_bytes(int B, int mode, int ck, int rt) {
  if (mode == kRope) return ceil_div(B, 8) * 8 * (8 + 32) * 4;
  return ck > 1 ? (rt * B + ck - 1) / ck * ck * 128 : 0;
}

// logits: an fp32 result, as the product over the vocabulary has it
inline LinearShape linear_shape(int B, int N, int K, int mode, int sms, bool logits) {
  LinearShape s{};
  if (K % kBlk != 0 || K < kBlk || B < 1 || B > 32 || N < 1) return s;
  const int tok = ceil_div(B, 8) * 8, blocks = K / kBlk;
  s.tk = linear_groups(N, K);
  if (mode == kStore && s.tk == 1) mode = kStream;
  s.tiles = mode == kGeglu ? ceil_div(N / 2, 16) : ceil_div(N, kTileRows);
  auto fit = [&](int kg, int ck, int rt, int stages) {
    s.kg = kg; s.ck = ck; s.rt = rt; s.stages = stages;
    int widest = 0;
    for (int r = 0; r < ck; r++) widest = std::max(widest, blocks * (r * kg + kg) / s.tk - blocks * (r * kg) / s.tk);
    if (s.sliced) {  // [column][K], two columns to 128 bytes of banks
      s.x_pitch = (widest * kBlk + 127) / 128 * 128 + 64;
      s.side_off = ceil_div(B * kSlices, 8) * 8 * s.x_pitch;
      s.x_bytes = (s.side_off + B * 4 + 127) / 128 * 128;
    } else {
      s.x_pitch = (widest * kBlk * 2 + 127) / 128 * 128 + 16;
      s.side_off = tok * s.x_pitch;
      s.x_bytes = (s.side_off + (B <= kNormTokens && (mode == kGeglu || mode == kRope) ? kNormTokens * 2 * 16 * 4 : 0) + 127) / 128 * 128;
    }
    const int warps = kg * rt;
    const int sums = warps * kTileRows * (tok + 1) * 4;
    s.scale_off = std::max(s.x_bytes + warps * stages * kStageBytes, mode == kStream ? 16 * tok * 8 : (sums + 127) / 128 * 128);
    s.recv_off = s.scale_off + rt * kTileRows * 4;
    s.smem = s.recv_off + linear_recv_bytes(B, mode, ck, rt);
    return s.smem <= kSmemMax;
  };
  if (mode == kStream) {
    auto warps_that_fit = [&](bool sliced) {
      s.sliced = sliced;
      int rt = 16;
      while (rt >= 1 && !fit(1, 1, rt, kStreamStages)) rt /= 2;
      return rt;
    };
    auto rounds = [&](int rt) { return ceil_div(s.tiles, (long long)sms * rt); };
    const int rt = warps_that_fit(false), sliced_rt = logits && B <= kSlicedTokens ? warps_that_fit(true) : 0;
    // Eight tokens' slices leave room for 8 warps from K = 3008 on, 4 from 5056, 2 from 6080 and none from 6848; bf16 rows for 16 below 6144. A
    // round (a tile for every warp) takes 7.6 to 8.5 us per 1024 of K with 8 warps on slices and 13.9 to 14.3 with 16 on bf16, but still 7.0
    // and 6.6 with 4 and 2 on slices: so 8 warps for 16 up to 1.8 times the rounds, and no others. Eight tokens, slices against bf16: K = 3072,
    // N = 100000 (3 rounds and 2) 76.4 / 86.0 us, 262144 (7 and 4) 159.6 / 166.2, 75000 (2 and 1) 57.1 / 51.5, 4096 x 60000 (2 and 1) 72.9 / 57.7,
    // 5120 x 50000 (4 warps) 104.9 / 67.9, 6144 x 50000 (2 warps) 239 / 91.
    if (sliced_rt < 1 || !(sliced_rt >= rt || (sliced_rt == 8 && 5 * rounds(sliced_rt) < 9 * rounds(rt)))) warps_that_fit(false);
    if ((s.sliced ? sliced_rt : rt) < 1) return LinearShape{};
    s.grid = std::min(sms, ceil_div(s.tiles, s.rt));
    s.ok = true;
    return s;
  }
  const int stages = ceil_div(blocks, s.tk);  // every block of a warp has its own place
  if (stages > 64) return s;
  if (mode == kRope) {
    s.ok = s.tk <= 16 && s.tk * kRopeTokens >= tok && fit(s.tk, 1, 1, stages);
    s.grid = s.tiles;
    return s;
  }
  // The fewest blocks per cluster whose activations leave room and whose clusters are all resident at once (a second wave cost
  // 7 us): clusters do not cross a GPC, of which eight with 16 SMs are counted on.
  auto one_wave = [&]() {
    const int clusters = s.grid / s.ck, per_sm = std::max(1, std::min(2048 / (s.kg * s.rt * 32), kSmemMax / s.smem));
    return s.ck == 1 ? s.grid <= sms * per_sm : clusters <= 8 * (16 / s.ck) * std::min(per_sm, 2);
  };
  for (int pass = 0; pass < 2; pass++)
    for (int ck = 1; ck <= 8 && ck <= s.tk; ck *= 2) {
      const int kg = s.tk / ck;
      if (kg > 16) continue;
      int rt = std::max(1, std::min(ceil_div((long long)s.tiles * ck, sms), 16 / kg));
      while (rt > 1 && !fit(kg, ck, rt, stages)) rt--;
      for (; rt <= 16 / kg && fit(kg, ck, rt, stages); rt++) {
        s.grid = ceil_div(s.tiles, rt) * ck;
        if (pass == 0 && !one_wave()) continue;
        s.ok = true;
        return s;
      }
    }
  return LinearShape{};
}

}  // namespace tb200
