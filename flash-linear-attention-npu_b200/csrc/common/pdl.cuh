// Programmatic dependent launch: a kernel launched with launch_pdl() may become resident while the kernel in front of it in
// the stream is still running, as soon as every CTA of that one has called pdl_trigger() or left.  What a launch costs between
// two dependent kernels (2 to 4 us on a B200: drain, launch latency, prologue) then lies under the tail of the first.
//
// The rule that keeps this invisible to callers: a kernel launched this way calls pdl_wait() in every thread that touches global memory,
// before its first access (prefetches into L2, which is the point of coherence, may come earlier).  pdl_wait() returns when the
// kernels in front are complete and their writes visible; since those waited too, everything before them in the stream is complete as
// well, so it does not matter which of the kernels a buffer was last written or read by.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace fla {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// overlap = false: an ordinary launch of such a kernel, for streams that share the SMs with another one - CTAs that only wait for their
// predecessor would keep the other stream's work from SMs that are free.
template <class... P, class... A>
cudaError_t launch_after(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  return launch_after(true, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}

}  // namespace fla
