// Programmatic dependent launch: a kernel launched with launch_dependent() may be scheduled while the
// kernel before it in the stream is still draining; its blocks become resident as that kernel's blocks
// retire and stop at pdl_wait() until the predecessor has completed and its writes are visible. At a few
// dozen images per GPU a network is a chain of kernels of a few microseconds each, and the gap between two
// kernels (launch processing, grid start) is a large part of the step; this hides most of it.
//
// Rules that keep it correct:
// (1) Every kernel launched this way executes pdl_wait() in every thread, before any global-memory access: as its first
//     statement, or in the tensor-core kernels after the barriers and the tensor memory are set up, which touches
//     nothing outside the SM. Its completion then implies the predecessor's, and ordering stays transitive along the
//     stream.
// (2) pdl_trigger() only says "my successor may be scheduled", it orders nothing. It comes after pdl_wait(), and after
//     the block has its tensor memory: a __syncthreads() stands between the allocation, which one warp makes, and the
//     trigger, for which one thread counts as the block. Otherwise, with another stream's kernel on the SM, the
//     successor's blocks could get the columns that this kernel's block is still waiting for, and keep them while they
//     wait for this kernel.
// Kernels launched the ordinary way in between serialize fully, as before. NNABLA_B200_PDL=0 turns the attribute off
// (ordinary launches; the waits are no-ops).
//
// When to trigger is a matter of time only. A kernel with a large share of the SM's shared memory that triggers early
// has the successor's blocks become resident beside it; the SM then never drains, and a streaming kernel goes on with
// the little L1 that such a split leaves (its loads in flight live there): max-pooling behind the stem 280 us instead
// of 180, a batch-256 network 5.0 ms instead of 4.5. So the stem, the pixel-major convolutions and the int8
// convolutions with an fp32 NCHW result trigger early up to early_trigger() values; gemm.cuh while its tiles make one
// round; the weight gradient while it is small (four taps per task), gemm2.cuh never. The int8 convolutions whose
// result is codes or channel-last trigger early at any size: what follows them in a network is the next convolution.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>

namespace nb200 {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether a large-shared-memory kernel with this many result values should let its successor in before it ends: up to
// 16 MB, where the next launch's start is a tenth of the kernel.
__device__ __forceinline__ bool early_trigger(int64_t values) { return values <= (4 << 20); }

inline bool pdl_enabled() {
  static const bool on = []() {
    const char *e = std::getenv("NNABLA_B200_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                    Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

} // namespace nb200
