// Memory accesses that several kernels share: shared-memory addresses and 16-byte reads, asynchronous 16-byte copies, 16 bytes
// from any byte address, and four look-ups in a byte table.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tb200 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {  // zeros when not valid
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// 16 bytes from byte offset off of x (4-byte aligned, total bytes) in five aligned words, of which only those that hold bytes of
// the tensor are read; bytes past the end are undefined. I: index type.
template <typename I>
__device__ __forceinline__ uint4 load16_any(const int8_t* x, I off, I total) {
  const I w0 = off & ~(I)3;
  const uint32_t sh = (uint32_t)(off & 3) * 8;
  uint32_t w[5];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    w[i] = 0;
    const I at = w0 + 4 * i;
    if (at + 4 <= total) {
      w[i] = *reinterpret_cast<const uint32_t*>(x + at);
    } else {
      for (int j = 0; at + j < total; j++) w[i] |= (uint32_t)(uint8_t)x[at + j] << (8 * j);
    }
  }
  return make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh), __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
}

// A 256-entry table applied to the four bytes of a word; lut is indexed by the raw byte.
__device__ __forceinline__ uint32_t lut_word(const uint8_t* lut, uint32_t w) {
  const uint32_t b0 = lut[w & 0xff], b1 = lut[(w >> 8) & 0xff], b2 = lut[(w >> 16) & 0xff], b3 = lut[w >> 24];
  return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
}

}  // namespace tb200
