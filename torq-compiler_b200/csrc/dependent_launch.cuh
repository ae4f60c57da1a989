// Programmatic dependent launch: a kernel launched through launch_dependent() may be scheduled while the kernel
// before it in the stream is still running (its blocks take the SMs the predecessor's blocks leave, and its
// prologue - shared-memory setup, barrier and TMEM allocation, loads of constants - runs in the predecessor's
// tail). Such a kernel must call grid_dependency_wait() before it reads or writes anything the predecessor may
// write or read: the wait returns once the predecessor has completed and its writes are visible. Without the
// launch attribute both device calls do nothing. TB200_NO_PDL=1 launches everything fully serialised (A/B aid).
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>
#include <utility>

namespace tb200 {

__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel's blocks be scheduled as soon as every block of this one has called it (or exited).
__device__ __forceinline__ void grid_dependency_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline bool dependent_launch_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("TB200_NO_PDL");
    v = !(e && *e && *e != '0');
  }
  return v != 0;
}

// A kernel lets the next one in only after its own wait has returned (grid_dependency_wait before grid_dependency_release):
// releasing first let chains of short kernels stack up a dozen deep, holding the registers and block slots of the one that
// had work. Measured on one-image inferences (56 and 120 launches of a few microseconds): released first 269 and 313 us,
// released after the wait 256 and 287 us, fully serialised 274 and 393 us. Two kernels release first. The tcgen05 products
// (gemm_tcgen05): persistent blocks that hold an SM's shared memory until they end. And the decoder's norm (rmsnorm_row), whose few
// blocks hold next to nothing while the product behind it is made resident (8 steps of one sequence 6467 -> 5987 us); with the
// decoder's products releasing first as well, 32 sequences took 9677 us instead of 9333. Where the planner fuses norms, two of them
// never follow each other, so nothing stacks up; with TB200_NO_DECODER_FUSION=1 pairs do, which costs time and nothing else.
constexpr long long kDependentMinBlocks = 4 * 148;  // persistent kernels: tiles x 2 from which their tail is worth overlapping

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent_if(bool large, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                       cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = large && dependent_launch_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    Args&&... args) {
  return launch_dependent_if(true, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

// The same with clusters of `cluster` consecutive blocks (1 = none); fully serialised when not programmatic.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent_cluster(int cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                            bool programmatic, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = programmatic && dependent_launch_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace tb200
