// Chunk bookkeeping of a packed batch: exclusive prefix sums of ceil(length / 64), made where the sequence boundaries already
// are (two copies from pageable host memory took the host longer than everything else a packed call did on it).
#include "fla_b200_internal.h"

namespace fla {

// One warp walks the sequences 32 at a time: N is a batch of sequences (tens to a few thousand), so this is latency, not work.
// host (optional): pinned host memory that receives the boundaries in [1, n + 1] and then, in [0], `tag`.
__global__ void chunk_offsets_kernel(const int32_t* cu, int32_t* co, int n, int32_t* host, int32_t tag) {
  const int lane = threadIdx.x;
  if (host) {
    for (int i = lane; i <= n; i += 32) host[1 + i] = cu[i];
    __threadfence_system();
    __syncwarp();
    if (lane == 0) *const_cast<volatile int32_t*>(host) = tag;
  }
  int base = 0;
  if (lane == 0) co[0] = 0;
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    int x = i < n ? (cu[i + 1] - cu[i] + 63) / 64 : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += up;
    }
    if (i < n) co[i + 1] = base + x;
    base += __shfl_sync(0xffffffffu, x, 31);
  }
}

}  // namespace fla

extern "C" FLA_API int fla_b200_chunk_offsets(const fla_tensor_t* cu, const fla_tensor_t* co, void* stream) {
  return fla_b200_chunk_bounds(cu, co, nullptr, 0, stream);
}

extern "C" FLA_API int fla_b200_chunk_bounds(const fla_tensor_t* cu, const fla_tensor_t* co, int32_t* host, int32_t tag, void* stream) {
  if (!cu || !co || !cu->data || !co->data) return FLA_ERR_NULL;
  for (const fla_tensor_t* t : {cu, co}) {
    if (t->dtype != FLA_I32) return FLA_ERR_DTYPE;
    if (t->ndim != 1 || t->shape[0] < 2 || t->shape[0] != cu->shape[0]) return FLA_ERR_SHAPE;
    if (t->stride[0] != 1) return FLA_ERR_LAYOUT;
  }
  fla::chunk_offsets_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const int32_t*>(cu->data),
                                                                             static_cast<int32_t*>(co->data), int(cu->shape[0] - 1), host, tag);
  return fla::cuda_status(cudaGetLastError());
}
