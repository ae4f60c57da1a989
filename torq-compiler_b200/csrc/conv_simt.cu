// CUDA-core (dp4a) convolution kernels: the general path for any kernel size,
// stride, dilation, padding and channel count. The tensor-core path in
// gemm_tcgen05.cu takes over the shapes it supports; results are bit-identical.
//
// Arithmetic (torq_hl.conv2d, compiler/torq/Conversions/LinalgToTorqHL/Conv2DPattern.cpp:478-654):
//   acc = bias + sum (x - izp) * (w - wzp), taps outside the image hold izp.
// The kernel accumulates raw x*w with dp4a, staging izp bytes for outside taps, so
//   sum (x-izp)(w-wzp) = sum x*w - izp*sum(w) - wzp*sum(x) + K*izp*wzp
// with sums over ALL K taps; the izp terms are constants per output channel and
// arrive folded into ChanParams::bias. int32 wrap-around keeps this exact.
#include <algorithm>

#include "kernels.h"
#include "dependent_launch.cuh"
#include "device_memory.cuh"

namespace tb200 {

namespace {

constexpr int BM = 64;   // output pixels per block
constexpr int BN = 64;   // output channels per block
constexpr int BK = 32;   // K bytes per step
constexpr int KW4 = BK / 4;
constexpr int LDS = KW4 + 1;  // padded row (words) -> conflict-free column reads

template <bool IC4>
__global__ void __launch_bounds__(256) conv2d_simt_kernel(ConvArgs a) {
  __shared__ uint32_t As[BM][LDS];
  __shared__ uint32_t Bs[BN][LDS];

  const int tid = threadIdx.x;
  const int tx = tid & 15;   // pixel lane
  const int ty = tid >> 4;   // oc lane
  const long long P = (long long)a.N * a.OH * a.OW;
  const long long p_base = (long long)blockIdx.x * BM;
  const int oc_base = blockIdx.y * BN;

  // this thread stages word `lw` of pixels lp0 and lp0 + 32, and of oc rows lp0, lp0 + 32
  const int lw = tid & 7;
  const int lp0 = tid >> 3;
  int ih0[2], iw0[2];
  const int8_t* xin[2];
  bool pvalid[2];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    long long p = p_base + lp0 + 32 * r;
    pvalid[r] = p < P;
    long long pp = pvalid[r] ? p : 0;
    int ow = (int)(pp % a.OW);
    long long t = pp / a.OW;
    int oh = (int)(t % a.OH);
    int n = (int)(t / a.OH);
    ih0[r] = oh * a.stride_h - a.pad_t;
    iw0[r] = ow * a.stride_w - a.pad_l;
    xin[r] = a.x + (size_t)n * a.H * a.W * a.IC;
  }
  const uint32_t zp_byte = (uint32_t)(a.input_zp & 0xff);
  const uint32_t zp_word = zp_byte * 0x01010101u;

  int acc[4][4];
  int xsum[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    xsum[i] = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0;
  }

  for (int k0 = 0; k0 < a.Kpad; k0 += BK) {
    const int k = k0 + lw * 4;
    // ---- stage A (implicit im2col gather) ----
    if (IC4) {
      int tap = k / a.IC;
      int ic = k - tap * a.IC;
      int kh = tap / a.KW;
      int kw = tap - kh * a.KW;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        uint32_t v = 0;
        if (pvalid[r] && k < a.K) {
          int ih = ih0[r] + kh * a.dil_h;
          int iw = iw0[r] + kw * a.dil_w;
          if (ih >= 0 && ih < a.H && iw >= 0 && iw < a.W)
            v = *reinterpret_cast<const uint32_t*>(xin[r] + ((size_t)ih * a.W + iw) * a.IC + ic);
          else
            v = zp_word;
        }
        As[lp0 + 32 * r][lw] = v;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        uint32_t v = 0;
        if (pvalid[r]) {
#pragma unroll
          for (int b = 0; b < 4; b++) {
            int kk = k + b;
            uint32_t byte = 0;
            if (kk < a.K) {
              int tap = kk / a.IC;
              int ic = kk - tap * a.IC;
              int kh = tap / a.KW;
              int kw = tap - kh * a.KW;
              int ih = ih0[r] + kh * a.dil_h;
              int iw = iw0[r] + kw * a.dil_w;
              if (ih >= 0 && ih < a.H && iw >= 0 && iw < a.W)
                byte = (uint8_t)xin[r][((size_t)ih * a.W + iw) * a.IC + ic];
              else
                byte = zp_byte;
            }
            v |= byte << (8 * b);
          }
        }
        As[lp0 + 32 * r][lw] = v;
      }
    }
    // ---- stage B (packed weights, rows padded to Kpad with zeros) ----
#pragma unroll
    for (int r = 0; r < 2; r++) {
      int oc = oc_base + lp0 + 32 * r;
      uint32_t v = 0;
      if (oc < a.OC) v = *reinterpret_cast<const uint32_t*>(a.w + (size_t)oc * a.Kpad + k);
      Bs[lp0 + 32 * r][lw] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < KW4; kk++) {
      uint32_t av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) av[i] = As[tx + 16 * i][kk];
#pragma unroll
      for (int j = 0; j < 4; j++) bv[j] = Bs[ty * 4 + j][kk];
#pragma unroll
      for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = __dp4a((int)av[i], (int)bv[j], acc[i][j]);
      }
      if (a.weight_zp != 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) xsum[i] = __dp4a((int)av[i], 0x01010101, xsum[i]);
      }
    }
    __syncthreads();
  }

  // ---- epilogue: bias, per-channel rescale, zero point, clamp ----
  const int oc0 = oc_base + ty * 4;
  ChanParams cp[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (oc0 + j < a.OC) cp[j] = a.chan[oc0 + j];
    else cp[j] = ChanParams{};
  }
  const bool hi = a.hi_shift != 0;
  const bool vec_ok = ((a.OC & 3) == 0) && (oc0 + 3 < a.OC);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    long long p = p_base + tx + 16 * i;
    if (p >= P) continue;
    int q[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      int v = acc[i][j] - a.weight_zp * xsum[i] + cp[j].bias;
      q[j] = hi ? requant_cp<true>(v, cp[j], a.out_zp, a.clamp_min, a.clamp_max)
                : requant_cp<false>(v, cp[j], a.out_zp, a.clamp_min, a.clamp_max);
      if (a.lut) q[j] = __ldg(a.lut + q[j] + 128);
    }
    int8_t* o = a.out + (size_t)p * a.OC + oc0;
    if (vec_ok) {
      *reinterpret_cast<uint32_t*>(o) = pack4(q[0], q[1], q[2], q[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (oc0 + j < a.OC) o[j] = (int8_t)q[j];
    }
  }
}

// Few input channels (IC <= 4, K = KH*KW*IC <= 64), e.g. the 3x3x3 stem of an image
// network: a thread gathers the K patch bytes of kPix output pixels into registers once
// and runs every output channel against weights broadcast from shared memory, so each
// weight word read serves kPix pixels. Same arithmetic as conv2d_simt_kernel (izp staged
// for taps outside the image).
constexpr int kPix = 2;
// S333: the 3x3 window over 3 channels, with the tap arithmetic folded at compile time.
template <int KWORDS, bool S333>
__global__ void __launch_bounds__(128) conv2d_smallic_kernel(ConvArgs a) {
  extern __shared__ uint32_t w_s[];  // [OC][KWORDS]
  for (int i = threadIdx.x; i < a.OC * KWORDS; i += blockDim.x) {
    const int oc = i / KWORDS, kw = i - oc * KWORDS;
    w_s[i] = (kw * 4 < a.Kpad) ? *reinterpret_cast<const uint32_t*>(a.w + (size_t)oc * a.Kpad + kw * 4) : 0u;
  }
  __syncthreads();
  const long long P = (long long)a.N * a.OH * a.OW;
  // pixel i of this thread: block base + i * 128 + thread, so a warp's stores stay adjacent
  const long long p_base = (long long)blockIdx.x * (128 * kPix) + threadIdx.x;
  const uint32_t zp_byte = (uint32_t)(a.input_zp & 0xff);

  uint32_t patch[kPix][KWORDS];
#pragma unroll
  for (int px = 0; px < kPix; px++) {
    const long long p = p_base + px * 128;
    const long long pp = p < P ? p : 0;
    const int ow = (int)(pp % a.OW);
    long long t = pp / a.OW;
    const int oh = (int)(t % a.OH);
    const int n = (int)(t / a.OH);
    const int ih0 = oh * a.stride_h - a.pad_t, iw0 = ow * a.stride_w - a.pad_l;
    const int8_t* xin = a.x + (size_t)n * a.H * a.W * a.IC;
#pragma unroll
    for (int i = 0; i < KWORDS; i++) {
      uint32_t word = 0;
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int k = 4 * i + b;
        if (S333) {
          if (k < 27) {
            constexpr int kdiv3[28] = {0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 3, 4, 4, 4, 5, 5, 5, 6, 6, 6, 7, 7, 7, 8, 8, 8, 9};
            const int tap = kdiv3[k < 27 ? k : 27], ic = k - tap * 3;
            const int kh = kdiv3[tap], kw = tap - kh * 3;
            const int ih = ih0 + kh * a.dil_h, iw = iw0 + kw * a.dil_w;
            const uint32_t byte = (ih >= 0 && ih < a.H && iw >= 0 && iw < a.W)
                                      ? (uint32_t)(uint8_t)xin[((size_t)ih * a.W + iw) * 3 + ic]
                                      : zp_byte;
            word |= byte << (8 * b);
          }
        } else if (k < a.K) {
          const int tap = k / a.IC, ic = k - tap * a.IC;
          const int kh = tap / a.KW, kw = tap - kh * a.KW;
          const int ih = ih0 + kh * a.dil_h, iw = iw0 + kw * a.dil_w;
          const uint32_t byte = (ih >= 0 && ih < a.H && iw >= 0 && iw < a.W)
                                    ? (uint32_t)(uint8_t)xin[((size_t)ih * a.W + iw) * a.IC + ic]
                                    : zp_byte;
          word |= byte << (8 * b);
        }
      }
      patch[px][i] = word;
    }
  }
  const bool hi = a.hi_shift != 0;
  for (int oc0 = 0; oc0 < a.OC; oc0 += 4) {
    int q[kPix][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int oc = min(oc0 + j, a.OC - 1);
      int acc[kPix];
#pragma unroll
      for (int px = 0; px < kPix; px++) acc[px] = 0;
#pragma unroll
      for (int i = 0; i < KWORDS; i++) {
        const int w = (int)w_s[oc * KWORDS + i];
#pragma unroll
        for (int px = 0; px < kPix; px++) acc[px] = __dp4a((int)patch[px][i], w, acc[px]);
      }
      const ChanParams cp = a.chan[oc];
#pragma unroll
      for (int px = 0; px < kPix; px++)
      {
        q[px][j] = hi ? requant_cp<true>(acc[px] + cp.bias, cp, a.out_zp, a.clamp_min, a.clamp_max)
                      : requant_cp<false>(acc[px] + cp.bias, cp, a.out_zp, a.clamp_min, a.clamp_max);
        if (a.lut) q[px][j] = __ldg(a.lut + q[px][j] + 128);
      }
    }
#pragma unroll
    for (int px = 0; px < kPix; px++) {
      const long long p = p_base + px * 128;
      if (p >= P) continue;
      int8_t* o = a.out + (size_t)p * a.OC;
      if ((a.OC & 3) == 0) {
        *reinterpret_cast<uint32_t*>(o + oc0) = pack4(q[px][0], q[px][1], q[px][2], q[px][3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (oc0 + j < a.OC) o[oc0 + j] = (int8_t)q[px][j];
      }
    }
  }
}

// Convolutions over exactly 16 input channels (the first stages of detector backbones: large
// frames, few channels). A tap of one pixel is one 16-byte load; a thread gathers the TAPS taps
// of its output pixel once (input zero point for taps outside the frame) and runs them against
// every output channel's weights, broadcast from shared memory: 4 dp4a per tap and channel.
// Weight rows are Kpad bytes apart (K = TAPS * 16 is a multiple of 16, Kpad of 32).
template <int TAPS>
__global__ void __launch_bounds__(128) conv2d_c16_kernel(ConvArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  extern __shared__ uint4 w16[];  // [OC][TAPS]
  for (int i = threadIdx.x; i < a.OC * TAPS; i += blockDim.x) {
    const int oc = i / TAPS, t = i - oc * TAPS;
    w16[i] = *reinterpret_cast<const uint4*>(a.w + (size_t)oc * a.Kpad + t * 16);
  }
  __syncthreads();
  const long long P = (long long)a.N * a.OH * a.OW;
  const long long p = (long long)blockIdx.x * 128 + threadIdx.x;
  if (p >= P) return;
  const int ow = (int)(p % a.OW);
  const long long t0 = p / a.OW;
  const int oh = (int)(t0 % a.OH), n = (int)(t0 / a.OH);
  const int ih0 = oh * a.stride_h - a.pad_t, iw0 = ow * a.stride_w - a.pad_l;
  const int8_t* xin = a.x + (size_t)n * a.H * a.W * 16;
  const uint32_t zw = (uint32_t)(a.input_zp & 0xff) * 0x01010101u;
  uint4 tap[TAPS];
#pragma unroll
  for (int t = 0; t < TAPS; t++) {
    const int kh = t / a.KW, kw = t - kh * a.KW;
    const int ih = ih0 + kh * a.dil_h, iw = iw0 + kw * a.dil_w;
    tap[t] = (ih >= 0 && ih < a.H && iw >= 0 && iw < a.W)
                 ? __ldg(reinterpret_cast<const uint4*>(xin + ((size_t)ih * a.W + iw) * 16))
                 : make_uint4(zw, zw, zw, zw);
  }
  const bool hi = a.hi_shift != 0;
  int8_t* o = a.out + (size_t)p * a.OC;
  for (int oc0 = 0; oc0 < a.OC; oc0 += 4) {
    int q[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int oc = min(oc0 + j, a.OC - 1);
      int acc = 0;
#pragma unroll
      for (int t = 0; t < TAPS; t++) {
        const uint4 w = w16[oc * TAPS + t];
        acc = __dp4a((int)tap[t].x, (int)w.x, acc);
        acc = __dp4a((int)tap[t].y, (int)w.y, acc);
        acc = __dp4a((int)tap[t].z, (int)w.z, acc);
        acc = __dp4a((int)tap[t].w, (int)w.w, acc);
      }
      const ChanParams cp = a.chan[oc];
      q[j] = hi ? requant_cp<true>(acc + cp.bias, cp, a.out_zp, a.clamp_min, a.clamp_max)
                : requant_cp<false>(acc + cp.bias, cp, a.out_zp, a.clamp_min, a.clamp_max);
      if (a.lut) q[j] = __ldg(a.lut + q[j] + 128);
    }
    if ((a.OC & 3) == 0) {
      *reinterpret_cast<uint32_t*>(o + oc0) = pack4(q[0], q[1], q[2], q[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (oc0 + j < a.OC) o[oc0 + j] = (int8_t)q[j];
    }
  }
}

// The 3x3 window over 3 channels (the stem of an image network) with the compact 32-bit epilogue records, on warp-level matrix
// instructions. A thread gathers a pixel: a kernel row is 9 consecutive bytes of the input, three aligned words and two funnel shifts
// (pixels whose window leaves the image, or whose words would reach past the tensor, gather byte by byte with the input zero
// point outside). The 27 bytes, packed into 8 words, are a row of 32 of the product's left operand: the warp leaves its 32 rows in
// shared memory and reads them back as fragments (ldmatrix), a k32 instruction then gives 16 pixels x 8 channels. Fragment column f
// of instruction j is channel (W / 4) (f / 2) + 2 j + f % 2 of a group of W, so that a lane ends with W / 4 consecutive channels of a pixel.
// What bounds it: integer issue, a third of it the gathering, half the rescale. Before, with 7 dp4a per output and 64-bit divisions per
// pixel: 25 instructions per output, 256 x 224 x 224 -> 32 channels 133 us, 64 x 640 x 640 -> 16 channels with a table 183 us; here 82 and 134.
constexpr int kStemPix = 8;  // most pixels a thread gathers, one after the other
// W: channels per pass over the fragments (16 or 32). I: index type, 32 bits where every offset fits.
template <int EPI, bool LUT, int W, typename I>
__global__ void __launch_bounds__(128) conv2d_stem333_kernel(ConvArgs a, int pixels) {
  constexpr int NJ = W / 8, CH = W / 4;  // instructions per 16 pixels, channels a lane ends with
  __shared__ __align__(16) uint4 rows_s[4][64];  // [warp][32 pixels x 2 halves]
  __shared__ uint8_t lut_s[LUT ? 256 : 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (LUT)
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut_s[LUT ? i : 0] = (uint8_t)a.lut[(int)(int8_t)i + 128];  // by the raw byte
  // weights and records of the first W channels (all of them in most stems)
  uint2 b[NJ];
  int4 q[CH];
  auto constants = [&](int oc0) {
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(a.w + (size_t)(oc0 + CH * (g >> 1) + 2 * j + (g & 1)) * a.Kpad) + t;
      b[j] = make_uint2(__ldg(w), __ldg(w + 4));
    }
#pragma unroll
    for (int c = 0; c < CH; c++) q[c] = __ldg(a.q4 + oc0 + CH * t + c);
  };
  constants(0);
  grid_dependency_wait();
  grid_dependency_release();
  if (LUT) __syncthreads();
  const I P = (I)a.N * a.OH * a.OW;
  I p0 = ((I)blockIdx.x * 4 + warp) * (32 * pixels);  // the warp's pixels
  if (p0 >= P) return;
  // this lane's pixel
  int ow, oh, n;
  {
    const I p = p0 + lane < P ? p0 + lane : 0, r = p / (I)a.OW;
    ow = (int)(p - r * (I)a.OW);
    n = (int)(r / (I)a.OH);
    oh = (int)(r - (I)n * a.OH);
  }
  const uint32_t zp_byte = (uint32_t)(a.input_zp & 0xff);
  const uint32_t lo2 = (uint32_t)(a.clamp_min & 0xffff) * 0x10001u, hi2 = (uint32_t)(a.clamp_max & 0xffff) * 0x10001u;
  const I row_bytes = (I)a.W * 3;
  uint4* mine = rows_s[warp];
  const uint32_t base = smem_u32(mine);
  const int swap = lane >> 2 & 1;  // half h of row r lies at 2 r + (h ^ (r >> 2 & 1)): eight rows' halves in different banks
  const uint32_t frag = base + (uint32_t)(2 * (lane & 15) + ((lane >> 4) ^ swap)) * 16;
  // the three words of each kernel row of the lane's pixel, asked for a pixel ahead
  uint32_t word[3][3], sh[3];
  bool inside;
  int ih0, iw0;
  auto ask = [&]() {
    ih0 = oh * a.stride_h - a.pad_t;
    iw0 = ow * a.stride_w - a.pad_l;
    const I off0 = (((I)n * a.H + ih0) * a.W + iw0) * 3;
    inside = ih0 >= 0 && ih0 + 2 < a.H && iw0 >= 0 && iw0 + 2 < a.W && ((off0 + 2 * row_bytes) & ~(I)3) + 12 <= (I)a.x_bytes;
    if (!inside) return;
#pragma unroll
    for (int kh = 0; kh < 3; kh++) {
      const I off = off0 + kh * row_bytes;
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(a.x + (off & ~(I)3));
#pragma unroll
      for (int k = 0; k < 3; k++) word[kh][k] = __ldg(wp + k);
      sh[kh] = (uint32_t)(off & 3) * 8;
    }
  };
  ask();
  for (int px = 0; px < pixels && p0 < P; px++, p0 += 32) {
    uint32_t row[3][3];  // per kernel row: bytes 0-3, 4-7, 8 (upper bytes of the third word are not used)
    if (inside) {
#pragma unroll
      for (int kh = 0; kh < 3; kh++) {
        row[kh][0] = __funnelshift_r(word[kh][0], word[kh][1], sh[kh]);
        row[kh][1] = __funnelshift_r(word[kh][1], word[kh][2], sh[kh]);
        row[kh][2] = word[kh][2] >> sh[kh];
      }
    } else {
      const int8_t* xin = a.x + (size_t)n * a.H * a.W * 3;
#pragma unroll
      for (int kh = 0; kh < 3; kh++) {
        const int ih = ih0 + kh;
        uint32_t c[9];
#pragma unroll
        for (int j = 0; j < 9; j++) {
          const int iw = iw0 + j / 3;
          c[j] = (ih >= 0 && ih < a.H && iw >= 0 && iw < a.W) ? (uint32_t)(uint8_t)xin[((size_t)ih * a.W + iw) * 3 + j % 3] : zp_byte;
        }
        row[kh][0] = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
        row[kh][1] = c[4] | (c[5] << 8) | (c[6] << 16) | (c[7] << 24);
        row[kh][2] = c[8];
      }
    }
    // K order (kh, kw, ic): bytes 0-8 row 0, 9-17 row 1, 18-26 row 2, bytes 27-31 meet zero weights
    mine[2 * lane + swap] = make_uint4(row[0][0], row[0][1], __byte_perm(row[0][2], row[1][0], 0x6540), __funnelshift_r(row[1][0], row[1][1], 24));
    mine[2 * lane + (swap ^ 1)] = make_uint4(__byte_perm(row[1][1], __byte_perm(row[1][2], row[2][0], 0x5400), 0x7653), __funnelshift_r(row[2][0], row[2][1], 16),
                                             __byte_perm(row[2][1], row[2][2], 0x0432), 0u);
    // the next pixel of this lane; behind the last one: read, never stored
    for (ow += 32; ow >= a.OW;) {
      ow -= a.OW;
      if (++oh == a.OH) {
        oh = 0;
        n++;
      }
    }
    if (p0 + 32 + lane >= P) ow = oh = n = 0;
    ask();
    __syncwarp();
    uint32_t f[2][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                   : "=r"(f[m][0]), "=r"(f[m][1]), "=r"(f[m][2]), "=r"(f[m][3]) : "r"(frag + m * 512) : "memory");
    __syncwarp();  // read before the next pixels are written
    const bool all = p0 + 32 <= P;
    int8_t* out = a.out + (size_t)(p0 + g) * a.OC + CH * t;
    for (int oc0 = 0; oc0 < a.OC; oc0 += W, out += W) {
      if (a.OC > W) constants(oc0);
      int8_t* o = out;
#pragma unroll
      for (int m = 0; m < 2; m++) {
        int acc[NJ][4];
#pragma unroll
        for (int j = 0; j < NJ; j++)
          asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                       : "=r"(acc[j][0]), "=r"(acc[j][1]), "=r"(acc[j][2]), "=r"(acc[j][3])
                       : "r"(f[m][0]), "r"(f[m][1]), "r"(f[m][2]), "r"(f[m][3]), "r"(b[j].x), "r"(b[j].y), "r"(0));
#pragma unroll
        for (int h = 0; h < 2; h++, o += 8 * a.OC) {
          uint32_t res[CH / 4];
#pragma unroll
          for (int k = 0; k < CH / 4; k++) {
            int r[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
              const int v = acc[2 * k + (c >> 1)][2 * h + (c & 1)];
              r[c] = EPI == 1 ? scale_q4_sign(v, q[4 * k + c]) : scale_q4(v, q[4 * k + c]);
            }
            res[k] = clamp_pack4(r[0], r[1], r[2], r[3], lo2, hi2);
            if (LUT) res[k] = lut_word(lut_s, res[k]);
          }
          if (all || p0 + 16 * m + 8 * h + g < P) {
            if (CH == 8) *reinterpret_cast<uint2*>(o) = make_uint2(res[0], res[CH / 4 - 1]);
            else *reinterpret_cast<uint32_t*>(o) = res[0];
          }
        }
      }
    }
  }
}

// The same at stride 2 on rows of whole words (a width that is a multiple of 4): no pixel is gathered. A warp takes 32 pixels of a result
// row: three kernel rows of 50 words, loaded as they lie (every word is inside the frame or outside), left in shared memory and read
// back as fragments. Windows of pixels two apart start 12 bytes apart, so the even pixels are one 16-row operand and the odd ones another, each
// with the weights at its own byte shift: nine words of K, a k32 and a k16 instruction. The words of the next 32 pixels are on their way
// while these are multiplied and rescaled. At the sizes above 70 and 107 us (14 instructions per output, half of the issue slots used by the 16
// warps that fit; limits of 96 and 80 registers spill and make the classifier 10 and 23 us slower), one frame of 640 x 640 7.7 -> 5.3 us.
template <int EPI, bool LUT, int W>
__global__ void __launch_bounds__(128, 4) conv2d_stem333_s2_kernel(ConvArgs a, int tiles, int tiles_x, int per_warp) {
  constexpr int NJ = W / 8, CH = W / 4;  // as above
  constexpr int kWords = 50, kPitch = 56;
  __shared__ uint32_t rows_s[4][3 * kPitch];
  __shared__ uint32_t w_s[2 * NJ * 3 * 32];  // [even / odd][instruction][word t, word t + 4, word 8][lane]
  __shared__ uint8_t lut_s[LUT ? 256 : 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int oc0 = blockIdx.y * W;
  const int sb = -3 * a.pad_l;  // first byte of the window of pixel 0; 32 pixels on is 192 bytes on
  if (LUT)
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut_s[LUT ? i : 0] = (uint8_t)a.lut[(int)(int8_t)i + 128];
  for (int i = threadIdx.x; i < 2 * NJ * 3 * 32; i += blockDim.x) {
    const int l = i & 31, k = (i >> 5) % 3, j = (i >> 5) / 3 % NJ, odd = (i >> 5) / (3 * NJ);
    const int word = k == 2 ? 8 : (l & 3) + 4 * k, kh = word / 3, first = 4 * (word % 3) - ((sb + 6 * odd) & 3);
    const int8_t* w = a.w + (size_t)(oc0 + CH * (l >> 3) + 2 * j + (l >> 2 & 1)) * a.Kpad + 9 * kh;
    uint32_t v = 0;
    for (int e = 0; e < 4; e++)
      if (first + e >= 0 && first + e < 9 && (k < 2 || (l & 3) == 0)) v |= (uint32_t)(uint8_t)w[first + e] << (8 * e);
    w_s[i] = v;
  }
  int4 q[CH];
#pragma unroll
  for (int c = 0; c < CH; c++) q[c] = __ldg(a.q4 + oc0 + CH * t + c);
  __syncthreads();
  uint32_t b[2][NJ][3];
#pragma unroll
  for (int o = 0; o < 2; o++)
#pragma unroll
    for (int j = 0; j < NJ; j++)
#pragma unroll
      for (int k = 0; k < 3; k++) b[o][j][k] = w_s[((o * NJ + j) * 3 + k) * 32 + lane];
  grid_dependency_wait();
  grid_dependency_release();
  int tile = (blockIdx.x * 4 + warp) * per_warp;
  const int last = min(tiles, tile + per_warp);
  if (tile >= last) return;
  int r = tile / tiles_x, tx = tile - r * tiles_x;  // r: result row over all images
  int n = r / a.OH, oh = r - n * a.OH;
  const uint32_t zp_word = (uint32_t)(a.input_zp & 0xff) * 0x01010101u;
  const uint32_t lo2 = (uint32_t)(a.clamp_min & 0xffff) * 0x10001u, hi2 = (uint32_t)(a.clamp_max & 0xffff) * 0x10001u;
  const int row_bytes = a.W * 3;
  uint32_t word[3][2];
  auto ask = [&]() {
    const int ih0 = oh * 2 - a.pad_t, col = (sb & ~3) + tx * 192 + 4 * lane;
#pragma unroll
    for (int kh = 0; kh < 3; kh++) {
      const bool row_ok = (unsigned)(ih0 + kh) < (unsigned)a.H;
      const int8_t* row = a.x + ((n * a.H + ih0 + kh) * row_bytes + col);
      word[kh][0] = word[kh][1] = zp_word;
      if (row_ok && (unsigned)col < (unsigned)row_bytes) word[kh][0] = __ldg(reinterpret_cast<const uint32_t*>(row));
      if (row_ok && lane < kWords - 32 && (unsigned)(col + 128) < (unsigned)row_bytes) word[kh][1] = __ldg(reinterpret_cast<const uint32_t*>(row + 128));
    }
  };
  ask();
  uint32_t* mine = rows_s[warp];
  // where this lane's words of the even pixel 2 g lie: word t, word t + 4, word 8 of its window
  auto at = [&](int w) { return mine + 3 * g + w / 3 * kPitch + w % 3; };
  const uint32_t* const f0 = at(t);
  const uint32_t* const f1 = at(t + 4);
  const uint32_t* const f2 = at(8);
  const int odd_words = ((sb & 3) + 6) >> 2;
  for (; tile < last; tile++) {
#pragma unroll
    for (int kh = 0; kh < 3; kh++) {
      mine[kh * kPitch + lane] = word[kh][0];
      if (lane < kWords - 32) mine[kh * kPitch + 32 + lane] = word[kh][1];
    }
    int8_t* out = a.out + ((size_t)(r * a.OW + tx * 32 + 2 * g) * a.OC + oc0 + CH * t);
    const int left = a.OW - tx * 32 - 2 * g;  // pixels from this lane's first on
    if (++tx == tiles_x) {
      tx = 0;
      r++;
      if (++oh == a.OH) {
        oh = 0;
        n++;
      }
    }
    if (tile + 1 < last) ask();
    __syncwarp();
    uint32_t f[2][6];
#pragma unroll
    for (int o = 0; o < 2; o++) {
      const int d = o ? odd_words : 0;
      f[o][0] = f0[d]; f[o][1] = f0[d + 24]; f[o][2] = f1[d]; f[o][3] = f1[d + 24]; f[o][4] = f2[d]; f[o][5] = f2[d + 24];
    }
    __syncwarp();  // read before the next rows are written
#pragma unroll
    for (int o = 0; o < 2; o++) {
      int acc[NJ][4];
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                     : "=r"(acc[j][0]), "=r"(acc[j][1]), "=r"(acc[j][2]), "=r"(acc[j][3])
                     : "r"(f[o][0]), "r"(f[o][1]), "r"(f[o][2]), "r"(f[o][3]), "r"(b[o][j][0]), "r"(b[o][j][1]), "r"(0));
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                     : "+r"(acc[j][0]), "+r"(acc[j][1]), "+r"(acc[j][2]), "+r"(acc[j][3])
                     : "r"(f[o][4]), "r"(f[o][5]), "r"(b[o][j][2]));
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {  // pixels 2 (g + 8 h) + o
        uint32_t res[CH / 4];
#pragma unroll
        for (int k = 0; k < CH / 4; k++) {
          int v[4];
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const int sum = acc[2 * k + (c >> 1)][2 * h + (c & 1)];
            v[c] = EPI == 1 ? scale_q4_sign(sum, q[4 * k + c]) : scale_q4(sum, q[4 * k + c]);
          }
          res[k] = clamp_pack4(v[0], v[1], v[2], v[3], lo2, hi2);
          if (LUT) res[k] = lut_word(lut_s, res[k]);
        }
        if (16 * h + o < left) {
          int8_t* p = out + (16 * h + o) * a.OC;
          if (CH == 8) *reinterpret_cast<uint2*>(p) = make_uint2(res[0], res[CH / 4 - 1]);
          else *reinterpret_cast<uint32_t*>(p) = res[0];
        }
      }
    }
  }
}

// FullyConnected on at most MR rows: one warp per output channel. The row(s) of x sit in shared memory (K bytes each);
// a lane takes 16 weights per step with one 16-byte load and runs them against the staged activations with dp4a;
// the warp adds its lanes' sums and lane 0 applies the exact rescale. Weights are read once, coalesced: HBM-bound.
template <int MR>
__global__ void __launch_bounds__(256) fc_rows_kernel(FcRowsArgs a) {
  extern __shared__ __align__(16) int8_t fc_x[];  // [MR][K]
  for (int i = threadIdx.x * 16; i < MR * a.K; i += blockDim.x * 16) {
    const int m = i / a.K, k = i - m * a.K;
    *reinterpret_cast<uint4*>(fc_x + i) = m < a.M ? *reinterpret_cast<const uint4*>(a.x + (size_t)m * a.K + k) : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * 8 + warp;
  if (n >= a.N) return;
  const int8_t* wrow = a.w + (size_t)n * a.K;
  int acc[MR];
#pragma unroll
  for (int m = 0; m < MR; m++) acc[m] = 0;
#pragma unroll 4
  for (int k = lane * 16; k < a.K; k += 32 * 16) {
    const uint4 wv = __ldg(reinterpret_cast<const uint4*>(wrow + k));
#pragma unroll
    for (int m = 0; m < MR; m++) {
      const uint4 xv = *reinterpret_cast<const uint4*>(fc_x + m * a.K + k);
      acc[m] = __dp4a((int)xv.x, (int)wv.x, acc[m]);
      acc[m] = __dp4a((int)xv.y, (int)wv.y, acc[m]);
      acc[m] = __dp4a((int)xv.z, (int)wv.z, acc[m]);
      acc[m] = __dp4a((int)xv.w, (int)wv.w, acc[m]);
    }
  }
#pragma unroll
  for (int m = 0; m < MR; m++)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
  if (lane == 0) {
    const ChanParams cp = a.chan[n];
#pragma unroll
    for (int m = 0; m < MR; m++)
      if (m < a.M) {
        int q = a.hi_shift ? requant_cp<true>(acc[m] + cp.bias, cp, a.out_zp, a.clamp_min, a.clamp_max)
                           : requant_cp<false>(acc[m] + cp.bias, cp, a.out_zp, a.clamp_min, a.clamp_max);
        if (a.lut) q = __ldg(a.lut + q + 128);
        a.out[(size_t)m * a.N + n] = (int8_t)q;
      }
  }
}

// Conv2D i16 x i8 (TB200_OP_CONV2D_I16): one thread per output; consecutive threads take consecutive output channels
// of a pixel, so the pixel's input window is read by the whole group and the weights stream per thread. 64-bit
// accumulation (TOSA's 48-bit accumulator never leaves it), then apply_scale_16:
// (acc * multiplier + 2^(shift-1)) >> shift, + out_zp, clamp, int16.
__global__ void __launch_bounds__(256) conv2d_i16_kernel(ConvI16Args a) {
  const long long total = (long long)a.N * a.OH * a.OW * a.OC;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int oc = (int)(idx % a.OC);
  long long p = idx / a.OC;
  const int ow = (int)(p % a.OW);
  p /= a.OW;
  const int oh = (int)(p % a.OH);
  const int n = (int)(p / a.OH);
  long long acc = a.bias[oc];
  const int8_t* wrow = a.w + (size_t)oc * a.KH * a.KW * a.IC;
  for (int kh = 0; kh < a.KH; kh++) {
    const int ih = oh * a.stride_h - a.pad_t + kh * a.dil_h;
    if (ih < 0 || ih >= a.H) continue;
    for (int kw = 0; kw < a.KW; kw++) {
      const int iw = ow * a.stride_w - a.pad_l + kw * a.dil_w;
      if (iw < 0 || iw >= a.W) continue;
      const int16_t* px = a.x + (((size_t)n * a.H + ih) * a.W + iw) * a.IC;
      const int8_t* wt = wrow + ((size_t)kh * a.KW + kw) * a.IC;
      int part = 0;  // |(x - zp) * (w - wzp)| < 2^16 * 2^8: 64 terms fit in 31 bits
      for (int c = 0; c < a.IC; c++) {
        part += ((int)px[c] - a.input_zp) * ((int)wt[c] - a.weight_zp);
        if ((c & 63) == 63) {
          acc += part;
          part = 0;
        }
      }
      acc += part;
    }
  }
  const int sh = a.shift[oc];
  long long r = ((acc * (long long)a.mult[oc] + (1ll << (sh - 1))) >> sh) + a.out_zp;
  r = r < a.clamp_min ? a.clamp_min : (r > a.clamp_max ? a.clamp_max : r);
  a.out[idx] = (int16_t)r;
}

}  // namespace

static bool conv_c16_applies(const ConvArgs& a) {
  const int taps = a.KH * a.KW;
  return a.IC == 16 && a.weight_zp == 0 && a.OC <= 256 && (taps == 9 || taps == 1 || taps == 25);
}

// the 3x3x3 stem with 32-bit epilogue records, output channels in whole 16-byte groups
static bool conv_stem333_shape(const ConvArgs& a) {
  return a.IC == 3 && a.KH == 3 && a.KW == 3 && a.dil_h == 1 && a.dil_w == 1 && a.weight_zp == 0 && a.epi != 0 &&
         (a.OC & 15) == 0 && a.OC <= 256;
}
static bool conv_stem333_applies(const ConvArgs& a) {
  return conv_stem333_shape(a) && a.q4 && ((uintptr_t)a.x & 3) == 0 && ((uintptr_t)a.out & 15) == 0;
}

const char* conv2d_simt_kernel_name(const ConvArgs& a) {
  if (conv_c16_applies(a)) return "conv2d_c16_dp4a";
  if (conv_stem333_shape(a)) return "conv2d_stem333_mma";
  return (a.IC <= 4 && a.K <= 64 && a.OC <= 256 && a.weight_zp == 0) ? "conv2d_smallic_dp4a" : "conv2d_simt";
}

void launch_conv2d_simt(const ConvArgs& a, cudaStream_t stream) {
  long long P = (long long)a.N * a.OH * a.OW;
  if (conv_c16_applies(a)) {
    const unsigned blocks = (unsigned)((P + 127) / 128);
    const int taps = a.KH * a.KW;
    const size_t smem = (size_t)a.OC * taps * 16;
    if (taps == 9) {
      launch_dependent(conv2d_c16_kernel<9>, dim3(blocks), dim3(128), smem, stream, a);
    } else if (taps == 1) {
      launch_dependent(conv2d_c16_kernel<1>, dim3(blocks), dim3(128), smem, stream, a);
    } else {
      static std::atomic<unsigned long long> attr{0};  // function attributes are per device
      if (first_use_on_device(attr)) {
        cudaFuncSetAttribute(conv2d_c16_kernel<25>, cudaFuncAttributeMaxDynamicSharedMemorySize, 256 * 25 * 16);
        mark_used_on_device(attr);
      }
      launch_dependent(conv2d_c16_kernel<25>, dim3(blocks), dim3(128), smem, stream, a);
    }
    return;
  }
  if (conv_stem333_applies(a)) {
    const int sms = current_sm_count();
    // a frame or two: as many blocks as there is work for
    const int pixels = (int)std::max(1ll, std::min((long long)kStemPix, P / (128ll * sms * 6)));
    const unsigned blocks = (unsigned)((P + 128 * pixels - 1) / (128 * pixels));
    // 32-bit offsets where the last pixel of the last block still has one
    const bool small = P + 128 * kStemPix < (1ll << 31) && a.x_bytes < (1ll << 31) - 64;
    const bool words = a.stride_h == 2 && a.stride_w == 2 && (a.W & 3) == 0;
    const int tiles_x = (a.OW + 31) / 32, tiles = small && words ? a.N * a.OH * tiles_x : 0;
    const int per_warp = std::max(1, (tiles + sms * 4 * 4 - 1) / (sms * 4 * 4));  // one wave of blocks, their weights laid out once
    const dim3 tile_grid((unsigned)((tiles + 4 * per_warp - 1) / (4 * per_warp)));
#define TB200_STEM(EPI, LUT, W)                                                                                                       \
  do {                                                                                                                                \
    if (small && words)                                                                                                               \
      launch_dependent(conv2d_stem333_s2_kernel<EPI, LUT, W>, dim3(tile_grid.x, (unsigned)(a.OC / W)), dim3(128), 0, stream, a, tiles, tiles_x, per_warp); \
    else if (small) launch_dependent(conv2d_stem333_kernel<EPI, LUT, W, int>, dim3(blocks), dim3(128), 0, stream, a, pixels);         \
    else launch_dependent(conv2d_stem333_kernel<EPI, LUT, W, long long>, dim3(blocks), dim3(128), 0, stream, a, pixels);              \
  } while (0)
#define TB200_STEM_EPI(LUT, W)               \
  do {                                       \
    if (a.epi == 1) TB200_STEM(1, LUT, W);   \
    else TB200_STEM(2, LUT, W);              \
  } while (0)
    if (a.OC % 32 == 0) {
      if (a.lut) TB200_STEM_EPI(true, 32);
      else TB200_STEM_EPI(false, 32);
    } else {
      if (a.lut) TB200_STEM_EPI(true, 16);
      else TB200_STEM_EPI(false, 16);
    }
#undef TB200_STEM_EPI
#undef TB200_STEM
    return;
  }
  if (a.IC <= 4 && a.K <= 64 && a.OC <= 256 && a.weight_zp == 0) {
    const unsigned blocks = (unsigned)((P + 128 * kPix - 1) / (128 * kPix));
    const int kwords = (a.K + 3) / 4;
    if (a.IC == 3 && a.KH == 3 && a.KW == 3)
      conv2d_smallic_kernel<7, true><<<blocks, 128, (size_t)a.OC * 7 * 4, stream>>>(a);
    else if (kwords <= 3) conv2d_smallic_kernel<3, false><<<blocks, 128, (size_t)a.OC * 3 * 4, stream>>>(a);
    else if (kwords <= 7) conv2d_smallic_kernel<7, false><<<blocks, 128, (size_t)a.OC * 7 * 4, stream>>>(a);
    else if (kwords <= 9) conv2d_smallic_kernel<9, false><<<blocks, 128, (size_t)a.OC * 9 * 4, stream>>>(a);
    else conv2d_smallic_kernel<16, false><<<blocks, 128, (size_t)a.OC * 16 * 4, stream>>>(a);
    return;
  }
  dim3 grid((unsigned)((P + BM - 1) / BM), (unsigned)((a.OC + BN - 1) / BN));
  if ((a.IC & 3) == 0)
    conv2d_simt_kernel<true><<<grid, 256, 0, stream>>>(a);
  else
    conv2d_simt_kernel<false><<<grid, 256, 0, stream>>>(a);
}

void launch_fc_rows(const FcRowsArgs& a, cudaStream_t stream) {
  const unsigned blocks = (unsigned)((a.N + 7) / 8);
  if (a.M <= 1) fc_rows_kernel<1><<<blocks, 256, (size_t)a.K, stream>>>(a);
  else if (a.M <= 2) fc_rows_kernel<2><<<blocks, 256, (size_t)2 * a.K, stream>>>(a);
  else fc_rows_kernel<4><<<blocks, 256, (size_t)4 * a.K, stream>>>(a);
}

void launch_conv2d_i16(const ConvI16Args& a, cudaStream_t stream) {
  const long long total = (long long)a.N * a.OH * a.OW * a.OC;
  conv2d_i16_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(a);
}

}  // namespace tb200
