// Bandwidth-bound layer kernels: rescaled add/sub/mul, 256-entry table,
// standalone rescale (also the building block of a rescaled concat), 2x nearest
// resize. 128-bit accesses wherever the channel count allows; grids sized in
// whole multiples of the SM count with grid-stride loops.
#include <algorithm>

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

// ---- add / sub / mul in TOSA form (ElementWiseBinaryPattern.cpp:385-570, MulPattern.cpp:229-238) ----
// add / sub as one linear function of the two bytes: out = clamp((xa * 2^8 * ma + xb * 2^8 * mb + K) >> (32 + F)), the
// three roundings of the op absorbed in K. The planner takes this form only after it has compared it with the exact op on
// all 65536 operand pairs (binary_linear_form). Per output: two byte extracts, two multiply-adds and a quarter of the
// packing, against two 256-entry look-ups (two wavefronts each), a 64-bit or 4-cycle multiply-high and the rounding before:
// 12.8 M elements 19 -> 9.3 us, 51 M elements 48 -> 33 us (4.6 TB/s). Loads in flight and the integer pipe share the bound:
// long scoreboard leads, issue slots 47 %, ALU 53 %.
__global__ void __launch_bounds__(kThreads) binary_linear_kernel(BinaryArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  const uint32_t lo2 = (uint32_t)((a.clamp_min << a.lin_f) & 0xffff) * 0x10001u;
  const uint32_t hi2 = (uint32_t)(((a.clamp_max << a.lin_f) | ((1 << a.lin_f) - 1)) & 0xffff) * 0x10001u;
  const int up = 8 - a.lin_f;  // brings the integer part to the high byte of its 16-bit field
  auto one = [&](int xa, int xb) { return mad_wide_hi(xb, a.lin_mb, (long long)xa * (long long)a.lin_ma + a.lin_k); };
  auto word = [&](uint32_t wa, uint32_t wb) {
    const int h0 = one(sx8_shl8<0>(wa), sx8_shl8<0>(wb)), h1 = one(sx8_shl8<1>(wa), sx8_shl8<1>(wb)),
              h2 = one(sx8_shl8<2>(wa), sx8_shl8<2>(wb)), h3 = one(sx8_shl8<3>(wa), sx8_shl8<3>(wb));
    uint32_t p, q;
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(p) : "r"(h1), "r"(h0));
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(q) : "r"(h3), "r"(h2));
    // clamped first, so that the shift cannot carry the low field into the integer part of the high one
    p = min_s16x2(max_s16x2(p, lo2), hi2) << up;
    q = min_s16x2(max_s16x2(q, lo2), hi2) << up;
    return __byte_perm(p, q, 0x7531);
  };
  const long long nvec = a.n >> 4;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long i = tid; i < nvec; i += stride) {
    const uint4 va = reinterpret_cast<const uint4*>(a.a)[i];
    const uint4 vb = reinterpret_cast<const uint4*>(a.b)[i];
    reinterpret_cast<uint4*>(a.out)[i] = make_uint4(word(va.x, vb.x), word(va.y, vb.y), word(va.z, vb.z), word(va.w, vb.w));
  }
  for (long long i = (nvec << 4) + tid; i < a.n; i += stride) a.out[i] = (int8_t)word((uint8_t)a.a[i], (uint8_t)a.b[i]);
}

// Every other case (mul, or an add without an exact linear form). An int8 operand takes 256 values, so its input-side
// rescale is a 256-entry table (filled here by the same apply_scale_32, one entry per thread); the output rescale stays
// arithmetic: EPI 0 = 64-bit, 1 / 2 = the compact 32-bit record (common.cuh) with / without the sign term, chosen by the
// planner when it can bound |operand sum or product| (it evaluates the same two tables).
template <int EPI>
__global__ void __launch_bounds__(kThreads) binary_kernel(BinaryArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ int ta[256], tb[256];  // indexed by the raw byte
  {
    const bool dr = a.double_round != 0;
    const int v = (int)(int8_t)threadIdx.x;
    ta[threadIdx.x] = apply_scale_32((v - a.a_zp) * (1 << a.a_lshift), a.a_mult, a.a_shift, dr);
    tb[threadIdx.x] = apply_scale_32((v - a.b_zp) * (1 << a.b_lshift), a.b_mult, a.b_shift, dr);
  }
  __syncthreads();
  const bool dr = a.double_round != 0;
  auto one = [&](uint32_t xa, uint32_t xb) {
    const int ra = ta[xa], rb = tb[xb];
    const int v = a.kind == 0 ? ra + rb : a.kind == 1 ? ra - rb : ra * rb;
    if (EPI == 0) return requant(v, a.out_mult, a.out_shift, dr, a.out_zp, a.clamp_min, a.clamp_max);
    const int r = EPI == 1 ? scale_q4_sign(v, a.q4) : scale_q4(v, a.q4);  // the output zero point rides in the record
    return max(a.clamp_min, min(a.clamp_max, r));
  };
  const long long nvec = a.n >> 4;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long i = tid; i < nvec; i += stride) {
    uint4 va = reinterpret_cast<const uint4*>(a.a)[i];
    uint4 vb = reinterpret_cast<const uint4*>(a.b)[i];
    uint32_t wa[4] = {va.x, va.y, va.z, va.w};
    uint32_t wb[4] = {vb.x, vb.y, vb.z, vb.w};
    uint32_t wo[4];
#pragma unroll
    for (int w = 0; w < 4; w++) {
      int q[4];
#pragma unroll
      for (int j = 0; j < 4; j++) q[j] = one((wa[w] >> (8 * j)) & 0xff, (wb[w] >> (8 * j)) & 0xff);
      wo[w] = pack4(q[0], q[1], q[2], q[3]);
    }
    reinterpret_cast<uint4*>(a.out)[i] = make_uint4(wo[0], wo[1], wo[2], wo[3]);
  }
  for (long long i = (nvec << 4) + tid; i < a.n; i += stride)
    a.out[i] = (int8_t)one((uint8_t)a.a[i], (uint8_t)a.b[i]);
}

// ---- table: out = table[x + 128] (ExtractPattern.cpp:97-135) ----
__global__ void __launch_bounds__(kThreads) table_kernel(const int8_t* __restrict__ x,
                                                         const int8_t* __restrict__ table,
                                                         int8_t* __restrict__ out, long long n) {
  __shared__ uint8_t lut[256];
  // index by the raw byte: entry for byte b is table[(int8)b + 128]
  lut[threadIdx.x] = (uint8_t)table[(int)(int8_t)threadIdx.x + 128];
  grid_dependency_wait();
  grid_dependency_release();
  __syncthreads();
  const long long nvec = n >> 4;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long i = tid; i < nvec; i += stride) {
    const uint4 v = reinterpret_cast<const uint4*>(x)[i];
    reinterpret_cast<uint4*>(out)[i] = make_uint4(lut_word(lut, v.x), lut_word(lut, v.y), lut_word(lut, v.z), lut_word(lut, v.w));
  }
  for (long long i = (nvec << 4) + tid; i < n; i += stride) out[i] = (int8_t)lut[(uint8_t)x[i]];
}

// ---- concatenation along the channels (ConcatOpPattern: every operand rescaled to the result's scale) ----
// All operands of a chain in one launch that writes whole rows. Bound by memory: a copy per operand wrote pieces of 16 .. 256
// bytes of every row and paid a launch for each - the 38 copies of YOLOv8n took 388 us at 64 frames, 13 launches 221 us of this kernel
// alone and 135 us with the wide one below (128 us of HBM time). A thread
// has kConcatFlight units in flight; a unit's row comes from one 32-bit division.
constexpr int kConcatFlight = 4;
enum { kAsIs = 0, kTables = 1, kLinear = 2 };
// A rescale as one multiply-add with 16 fraction bits per byte, where the planner found one that gives the table exactly.
__device__ __forceinline__ uint4 rescale_linear(const uint4& v, int m, int k) {
  auto word = [&](uint32_t w) {
    const int q0 = (int)(int8_t)w * m + k, q1 = (int)(int8_t)(w >> 8) * m + k, q2 = (int)(int8_t)(w >> 16) * m + k, q3 = ((int)w >> 24) * m + k;
    return sat_pack4(q0 >> 16, q1 >> 16, q2 >> 16, q3 >> 16);
  };
  return make_uint4(word(v.x), word(v.y), word(v.z), word(v.w));
}
template <int MODE>
__global__ void __launch_bounds__(kThreads) concat_kernel(const __grid_constant__ ConcatArgs a) {
  constexpr bool LUT = MODE == kTables;
  __shared__ uint8_t lut[LUT ? kConcatMax : 1][256];
  if (LUT) {
    for (int o = 0; o < a.n; o++)
      if (a.lut[o]) lut[LUT ? o : 0][threadIdx.x] = a.lut[o][threadIdx.x];
    __syncthreads();
  }
  grid_dependency_wait();
  grid_dependency_release();
  const long long total = a.rows * a.row_units, stride = (long long)gridDim.x * kThreads;
  for (long long i0 = (long long)blockIdx.x * kThreads + threadIdx.x; i0 < total; i0 += kConcatFlight * stride) {
    uint4 v[kConcatFlight];
    int op[kConcatFlight];
#pragma unroll
    for (int u = 0; u < kConcatFlight; u++) {
      const long long i = i0 + u * stride;
      v[u] = make_uint4(0, 0, 0, 0);
      op[u] = 0;
      if (i < total) {
        long long r;
        if (total < (1ll << 32)) r = (uint32_t)i / (uint32_t)a.row_units;
        else r = i / a.row_units;
        const int c = (int)(i - r * a.row_units);
        const int8_t* x = a.x[0];
        int units = a.units[0], at = c;
#pragma unroll
        for (int o = 1; o < kConcatMax; o++)
          if (o < a.n && c >= a.first[o]) {
            x = a.x[o];
            units = a.units[o];
            at = c - a.first[o];
            op[u] = o;
          }
        v[u] = __ldcs(reinterpret_cast<const uint4*>(x) + r * units + at);
      }
    }
#pragma unroll
    for (int u = 0; u < kConcatFlight; u++) {
      const long long i = i0 + u * stride;
      if (i >= total) break;
      if (LUT && a.lut[op[u]]) {
        const uint8_t* t = lut[LUT ? op[u] : 0];
        v[u] = make_uint4(lut_word(t, v[u].x), lut_word(t, v[u].y), lut_word(t, v[u].z), lut_word(t, v[u].w));
      }
      if (MODE == kLinear && a.lin_m[op[u]] != 0) v[u] = rescale_linear(v[u], a.lin_m[op[u]], a.lin_k[op[u]]);
      reinterpret_cast<uint4*>(a.out)[i] = v[u];
    }
  }
}

// Large concatenations of operands in whole 32-byte sectors: blockIdx.y is the operand, whose units a block reads as they lie (no choice of
// the operand per unit); a unit's row comes from one multiplication. Operands of 16 channels stay above: halves of sectors from
// different blocks cost more than the choice (160 x 160 x three of 16: 55 us here, 43 above). The nine concatenations of the detector at 64 frames
// that copy 121 -> 67 us, three of those that rescale 56 -> 25 us.
template <bool LIN>
__global__ void __launch_bounds__(kThreads) concat_wide_kernel(const __grid_constant__ ConcatArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  const int o = blockIdx.y, units = a.units[o], m = LIN ? a.lin_m[o] : 0, k = LIN ? a.lin_k[o] : 0;
  const uint32_t total = (uint32_t)a.rows * (uint32_t)units, per_row = a.per_row[o];
  const uint4* x = reinterpret_cast<const uint4*>(a.x[o]);
  uint4* out = reinterpret_cast<uint4*>(a.out) + a.first[o];
  const uint32_t i0 = blockIdx.x * (kThreads * kConcatFlight) + threadIdx.x;
  uint4 v[kConcatFlight];
#pragma unroll
  for (int u = 0; u < kConcatFlight; u++)
    if (i0 + u * kThreads < total) v[u] = __ldcs(x + i0 + u * kThreads);
#pragma unroll
  for (int u = 0; u < kConcatFlight; u++) {
    const uint32_t i = i0 + u * kThreads;
    if (i >= total) break;
    if (LIN && m != 0) v[u] = rescale_linear(v[u], m, k);
    const uint32_t r = __umulhi(i, per_row);
    out[(size_t)r * a.row_units + (i - r * units)] = v[u];
  }
}

// ---- standalone rescale i8 -> i8 (PatternUtils.cpp:426-435,3441-3451) ----
__global__ void __launch_bounds__(kThreads) rescale_kernel(RescaleArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  const long long total = a.rows * a.C;
  const bool dr = a.double_round != 0;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    int c = (int)(idx % a.C);
    long long r = idx / a.C;
    ChanParams cp = a.chan[a.per_channel ? c : 0];
    int v = (int)a.x[idx] - a.input_zp;
    a.out[(size_t)r * a.out_row_stride + a.out_col_offset + c] =
        (int8_t)requant(v, cp.mult, cp.shift, dr, a.out_zp, a.clamp_min, a.clamp_max);
  }
}

// 16 channels per thread when the rows allow 16-byte accesses; IDENT: the rescale is a pass-through
// (multiplier 2^30, shift 30, equal zero points, full clamp range), i.e. a strided copy
template <bool IDENT>
__global__ void __launch_bounds__(kThreads) rescale_vec16_kernel(RescaleArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  const int cv = a.C >> 4;
  const long long total = a.rows * cv;
  const bool dr = a.double_round != 0;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int c16 = (int)(idx % cv);
    const long long r = idx / cv;
    uint4 v = __ldg(reinterpret_cast<const uint4*>(a.x + (size_t)r * a.C) + c16);
    if (!IDENT) {
      uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        int o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const ChanParams cp = a.chan[a.per_channel ? c16 * 16 + q * 4 + j : 0];
          o[j] = requant(sx8(w[q], j) - a.input_zp, cp.mult, cp.shift, dr, a.out_zp, a.clamp_min, a.clamp_max);
        }
        w[q] = pack4(o[0], o[1], o[2], o[3]);
      }
      v = make_uint4(w[0], w[1], w[2], w[3]);
    }
    *reinterpret_cast<uint4*>(a.out + (size_t)r * a.out_row_stride + a.out_col_offset + c16 * 16) = v;
  }
}

// Per-tensor constants: the rescale is a function of the input byte alone, so it runs as a 256-entry table
// in shared memory (one entry per thread, filled by the same requant), 16 channels per thread.
__global__ void __launch_bounds__(kThreads) rescale_lut_vec16_kernel(RescaleArgs a) {
  grid_dependency_wait();
  grid_dependency_release();
  __shared__ uint8_t lut[256];  // indexed by the raw byte
  {
    const ChanParams cp = a.chan[0];
    lut[threadIdx.x] = (uint8_t)requant((int)(int8_t)threadIdx.x - a.input_zp, cp.mult, cp.shift, a.double_round != 0,
                                        a.out_zp, a.clamp_min, a.clamp_max);
  }
  __syncthreads();
  const int cv = a.C >> 4;
  const long long total = a.rows * cv;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int c16 = (int)(idx % cv);
    const long long r = idx / cv;
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.x + (size_t)r * a.C) + c16);
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      uint32_t o = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) o |= (uint32_t)lut[(w[k] >> (8 * j)) & 0xff] << (8 * j);
      w[k] = o;
    }
    *reinterpret_cast<uint4*>(a.out + (size_t)r * a.out_row_stride + a.out_col_offset + c16 * 16) =
        make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// ---- nearest 2x (PatternUtils.cpp:489-491): out[y,x] = in[y/2, x/2] ----
__global__ void __launch_bounds__(kThreads) resize_nn2x_vec16_kernel(const int8_t* __restrict__ x, int8_t* __restrict__ out,
                                                                     int N, int H, int W, int C) {
  grid_dependency_wait();
  grid_dependency_release();
  const int cv = C >> 4;
  const long long total = (long long)N * 2 * H * 2 * W * cv;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int c16 = (int)(idx % cv);
    long long p = idx / cv;
    const int ow = (int)(p % (2 * W));
    long long t = p / (2 * W);
    const int oh = (int)(t % (2 * H));
    const int n = (int)(t / (2 * H));
    reinterpret_cast<uint4*>(out)[idx] =
        __ldg(reinterpret_cast<const uint4*>(x + (((size_t)n * H + (oh >> 1)) * W + (ow >> 1)) * C) + c16);
  }
}

__global__ void __launch_bounds__(kThreads) resize_nn2x_kernel(const int8_t* __restrict__ x,
                                                               int8_t* __restrict__ out, int N, int H,
                                                               int W, int C) {
  const long long total = (long long)N * 2 * H * 2 * W * C;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    int c = (int)(idx % C);
    long long p = idx / C;
    int ow = (int)(p % (2 * W));
    long long t = p / (2 * W);
    int oh = (int)(t % (2 * H));
    int n = (int)(t / (2 * H));
    out[idx] = x[(((size_t)n * H + (oh >> 1)) * W + (ow >> 1)) * C + c];
  }
}

}  // namespace

void launch_binary(const BinaryArgs& a, cudaStream_t stream) {
  if (a.lin) launch_dependent(binary_linear_kernel, dim3(grid_for((a.n + 15) / 16)), dim3(kThreads), 0, stream, a);
  else if (a.epi == 1) launch_dependent(binary_kernel<1>, dim3(grid_for((a.n + 15) / 16)), dim3(kThreads), 0, stream, a);
  else if (a.epi == 2) launch_dependent(binary_kernel<2>, dim3(grid_for((a.n + 15) / 16)), dim3(kThreads), 0, stream, a);
  else launch_dependent(binary_kernel<0>, dim3(grid_for((a.n + 15) / 16)), dim3(kThreads), 0, stream, a);
}

void launch_table(const int8_t* x, const int8_t* table, int8_t* out, long long n, cudaStream_t stream) {
  launch_dependent(table_kernel, dim3(grid_for((n + 15) / 16)), dim3(kThreads), 0, stream, x, table, out, n);
}

void launch_concat(const ConcatArgs& a, cudaStream_t stream) {
  bool lut = false;
  for (int o = 0; o < a.n; o++) lut |= a.lut[o] != nullptr;
  // from about four units a thread of a full chip on; the quotient by multiplication is exact below 2^32 / units
  ConcatArgs w = a;
  int widest = 0;
  bool linear = true, sectors = true;
  for (int o = 0; o < a.n; o++) {
    w.per_row[o] = (uint32_t)((0x100000000ull + a.units[o] - 1) / a.units[o]);
    widest = std::max(widest, a.units[o]);
    sectors = sectors && a.units[o] % 2 == 0;
    linear = linear && (!a.lut[o] || a.lin_m[o] != 0);
  }
  if (linear && sectors && a.rows * a.row_units >= 4ll * kThreads * 4 * current_sm_count() && a.rows * a.row_units < (1ll << 31) && a.rows * widest < (1ll << 32) / widest) {
    const dim3 wide((unsigned)((a.rows * widest + kThreads * kConcatFlight - 1) / (kThreads * kConcatFlight)), (unsigned)a.n);
    if (lut) launch_dependent(concat_wide_kernel<true>, wide, dim3(kThreads), 0, stream, w);
    else launch_dependent(concat_wide_kernel<false>, wide, dim3(kThreads), 0, stream, w);
    return;
  }
  const long long blocks = (a.rows * a.row_units + kThreads - 1) / kThreads, most = 8ll * current_sm_count();
  const dim3 grid((unsigned)(blocks < most ? blocks : most));
  if (lut && linear) launch_dependent(concat_kernel<kLinear>, grid, dim3(kThreads), 0, stream, a);
  else if (lut) launch_dependent(concat_kernel<kTables>, grid, dim3(kThreads), 0, stream, a);
  else launch_dependent(concat_kernel<kAsIs>, grid, dim3(kThreads), 0, stream, a);
}

void launch_rescale(const RescaleArgs& a, cudaStream_t stream) {
  const bool vec = (a.C & 15) == 0 && (a.out_row_stride & 15) == 0 && (a.out_col_offset & 15) == 0 &&
                   ((uintptr_t)a.x & 15) == 0 && ((uintptr_t)a.out & 15) == 0;
  if (vec && a.identity) launch_dependent(rescale_vec16_kernel<true>, dim3(grid_for(a.rows * (a.C >> 4))), dim3(kThreads), 0, stream, a);
  else if (vec && !a.per_channel) launch_dependent(rescale_lut_vec16_kernel, dim3(grid_for(a.rows * (a.C >> 4))), dim3(kThreads), 0, stream, a);
  else if (vec) launch_dependent(rescale_vec16_kernel<false>, dim3(grid_for(a.rows * (a.C >> 4))), dim3(kThreads), 0, stream, a);
  else launch_dependent(rescale_kernel, dim3(grid_for(a.rows * a.C)), dim3(kThreads), 0, stream, a);
}

void launch_resize_nn2x(const int8_t* x, int8_t* out, int N, int H, int W, int C, cudaStream_t stream) {
  if ((C & 15) == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)out & 15) == 0) {
    launch_dependent(resize_nn2x_vec16_kernel, dim3(grid_for((long long)N * 4 * H * W * (C >> 4))), dim3(kThreads), 0, stream, x, out, N, H, W, C);
    return;
  }
  resize_nn2x_kernel<<<grid_for((long long)N * 4 * H * W * C), kThreads, 0, stream>>>(x, out, N, H, W, C);
}

}  // namespace tb200
