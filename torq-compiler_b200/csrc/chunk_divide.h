// Division of a small count by a launch constant with one 32-bit multiplication and a shift: c / d = (c * ceil(2^s / d)) >> s for
// s = 18 + floor(log2 d). With ceil(2^s / d) = (2^s + e) / d and e < d the result is exact while c * e < 2^s, so for c < 2^18, and the
// product stays below 2^32 for c < 2^13. c is a 16-byte chunk of a small convolution's K axis, of which there are at most 4096
// and the three that fill its last step. (The high word of a product needs no s, but cost the detector at one frame 2.8 of 232.6 us;
// this form 0.1.)
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define TB200_BOTH __host__ __device__ __forceinline__
#else
#define TB200_BOTH inline
#endif

namespace tb200 {

constexpr int kMaxChunks = 4096;

struct ChunkDivisor {
  uint32_t inv;
  int shift;
};

inline ChunkDivisor chunk_divisor(int d) {
  int shift = 18;
  while ((d >> (shift - 18)) > 1) shift++;
  return {(uint32_t)(((1ull << shift) + (uint64_t)d - 1) / (uint64_t)d), shift};
}
TB200_BOTH int divide_chunk(int c, const ChunkDivisor& d) { return (int)(((uint32_t)c * d.inv) >> d.shift); }

// the same for a tap by the window's width: both at most kMaxTaps (and the three chunks of the last step that lie behind it)
constexpr int kMaxTaps = 64;
inline uint32_t tap_divisor(int kw) { return ((1u << 20) + (uint32_t)kw - 1) / (uint32_t)kw; }
TB200_BOTH int divide_tap(int tap, uint32_t inv) { return (int)(((uint32_t)tap * inv) >> 20); }

}  // namespace tb200
