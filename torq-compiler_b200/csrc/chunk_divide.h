// Division of a small count by a launch constant with one multiplication: c / d = floor(2c * ceil(2^31 / d) / 2^32). With
// ceil(2^31 / d) = (2^31 + e) / d and e < d the result is exact while c * e < 2^31, so for every c and d up to 2^15 - and c is a 16-byte
// chunk of a small convolution's K axis, of which there are at most 4096 and the three that fill its last step.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define TB200_BOTH __host__ __device__ __forceinline__
#else
#define TB200_BOTH inline
#endif

namespace tb200 {

constexpr int kMaxChunks = 4096;

TB200_BOTH uint32_t divide_constant(int d) { return ((1u << 31) + (uint32_t)d - 1) / (uint32_t)d; }
TB200_BOTH int divide_by(int c, uint32_t constant) { return (int)(((uint64_t)(2u * (uint32_t)c) * constant) >> 32); }

}  // namespace tb200
