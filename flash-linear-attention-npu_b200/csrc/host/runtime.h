// What every operator of the PyTorch binding needs between a Python call and a launch: tensor descriptors, the device check and
// guard, allocation, the two-phase call of the C ABI, and the status word.  The same duties as fla_b200/_runtime.py (which
// serves the stage operators through ctypes); there they cost 40 to 60 us per operator call on the host of a B200 node -
// more than the kernels of a decode step take - here about 5.
#pragma once
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <array>
#include <optional>
#include "../../../include/fla_b200.h"

namespace fla_host {

using at::Tensor;

// The entry points of libfla_b200.so, looked up once in the handle that fla_b200.load_library() opened.
#define FLA_HOST_FNS(X)                                                                                                    \
  X(recurrent_gdn_workspace_size) X(recurrent_gdn) X(causal_conv1d_fwd_workspace_size) X(causal_conv1d_fwd)                \
  X(causal_conv1d_bwd_workspace_size) X(causal_conv1d_bwd) X(causal_conv1d_update_workspace_size) X(causal_conv1d_update)  \
  X(gdn_chunk_fwd_workspace_size) X(gdn_chunk_segments_size) X(gdn_chunk_fwd) X(gdn_chunk_bwd_workspace_size) X(gdn_chunk_bwd)                        \
  X(kda_chunk_fwd_workspace_size) X(kda_chunk_fwd) X(kda_chunk_bwd_workspace_size) X(kda_chunk_bwd) X(kda_chunk_saved_size) \
  X(l2norm_fwd) X(l2norm_bwd) X(convert) X(chunk_offsets) X(chunk_bounds)
struct Library {
#define FLA_DECL(n) decltype(&fla_b200_##n) n = nullptr;
  FLA_HOST_FNS(FLA_DECL)
#undef FLA_DECL
};
extern Library lib;
extern bool check_status;     // read the device status word back after each call of an operator that has one

[[noreturn]] void fail(const char* op, int status);
inline void ok_or_throw(const char* op, int status) {
  if (status != FLA_OK) fail(op, status);
}

int32_t dtype_code(at::ScalarType t, const char* name);

// Null descriptor for an undefined tensor (argument absent).
inline fla_tensor_t desc(const Tensor& t, const char* name = "tensor") {
  fla_tensor_t d{};
  if (!t.defined()) return d;
  TORCH_CHECK(t.dim() <= FLA_MAX_DIMS, name, ": rank ", t.dim(), " exceeds ", FLA_MAX_DIMS);
  d.dtype = dtype_code(t.scalar_type(), name);
  d.data = t.numel() ? t.data_ptr() : nullptr;
  d.ndim = int32_t(t.dim());
  for (int i = 0; i < d.ndim; ++i) {
    d.shape[i] = t.size(i);
    d.stride[i] = t.stride(i);
  }
  return d;
}

// A dense tensor that is part of a larger allocation.
inline fla_tensor_t desc_at(void* data, at::ScalarType t, std::initializer_list<int64_t> sizes) {
  fla_tensor_t d{};
  d.data = data;
  d.dtype = dtype_code(t, "tensor");
  d.ndim = int32_t(sizes.size());
  int64_t stride = 1;
  for (int i = d.ndim - 1; i >= 0; --i) {
    d.shape[i] = sizes.begin()[i];
    d.stride[i] = stride;
    stride *= d.shape[i];
  }
  return d;
}

// All tensors of one call live on one CUDA device of the right architecture; there is no CPU path.
class Device {
 public:
  explicit Device(const char* op) : op_(op) {}
  Device& operator()(const Tensor& t) {
    if (!t.defined()) return *this;
    TORCH_CHECK(t.is_cuda(), op_, ": tensors must be on a CUDA device, got ", t.device(), " (no CPU fallback exists)");
    if (!set_) {
      dev_ = t.device();
      set_ = true;
    } else {
      TORCH_CHECK(t.device() == dev_, op_, ": all tensors must be on the same device, got ", dev_, " and ", t.device());
    }
    return *this;
  }
  at::Device get() const;      // also checks the architecture

 private:
  const char* op_;
  at::Device dev_{at::kCUDA, 0};
  bool set_ = false;
};

inline Tensor empty(at::IntArrayRef sizes, at::ScalarType t, at::Device d) {
  return Tensor(at::detail::empty_cuda(sizes, t, d, std::nullopt));
}
inline void* current_stream(at::Device d) { return c10::cuda::getCurrentCUDAStream(d.index()).stream(); }

void raise_device_status(const char* op, const Tensor& ws);

template <class A>
void two_phase(const char* op, int (*size)(const A*, uint64_t*), int (*run)(const A*, void*, uint64_t, void*), const A& a, at::Device d,
               bool has_status = false) {
  c10::cuda::CUDAGuard guard(d);
  uint64_t bytes = 0;
  if (int st = size(&a, &bytes)) fail((std::string(op) + " workspace query").c_str(), st);
  Tensor ws;      // goes back to the caching allocator in stream order at the end of this call
  if (bytes) ws = empty({int64_t(bytes)}, at::kByte, d);
  ok_or_throw(op, run(&a, bytes ? ws.data_ptr() : nullptr, bytes, current_stream(d)));
  if (has_status && check_status && bytes) raise_device_status(op, ws);
}
template <class... P, class... Q>
void one_phase(const char* op, at::Device d, int (*run)(P...), Q... args) {
  c10::cuda::CUDAGuard guard(d);
  ok_or_throw(op, run(args..., current_stream(d)));
}

// A dense copy of `t` in `dtype` by the library's conversion kernel.
Tensor convert(const Tensor& t, at::ScalarType dtype, const char* op);
// `t` in `dtype`, differentiable; `t` itself when it already has that dtype.
Tensor to_dtype(const Tensor& t, at::ScalarType dtype, const char* op);

// Kernels address tokens by one flat row index: batch rows must sit back to back, channels contiguous.
inline bool rows_ok(const Tensor& t) { return t.stride(-1) == 1 && (t.size(0) <= 1 || t.stride(0) == t.size(1) * t.stride(1)); }
inline Tensor as_rows(const Tensor& t) { return rows_ok(t) ? t : t.contiguous(); }

constexpr int64_t kChunk = 64;
// Chunk geometry of a batch: fixed-length rows, or a packed batch whose boundaries are read back from cu_seqlens.
struct Geometry {
  Tensor cu, co;                     // int32 [N + 1] on the device, undefined for fixed lengths
  int64_t N = 0, max_len = 0, chunks = 0;
};
Geometry geometry(const char* op, int64_t B, int64_t T, const Tensor& cu_seqlens, at::Device d);

inline bool any_requires_grad(std::initializer_list<Tensor> ts) {
  for (const Tensor& t : ts)
    if (t.defined() && t.requires_grad()) return true;
  return false;
}

// Arguments of an autograd node that may be absent: an undefined tensor is not a valid input of one.
using OptTensor = std::optional<Tensor>;
inline OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }
inline Tensor value(const OptTensor& t) { return t ? *t : Tensor(); }

// ---- operators (conv.cpp, recurrent.cpp, gdn.cpp, kda.cpp)
using Pair = std::pair<Tensor, Tensor>;
Pair l2norm_fwd(const Tensor& x, double eps, std::optional<at::ScalarType> out);
Tensor l2norm_bwd(const Tensor& y, const Tensor& rstd, const Tensor& dy, double eps, std::optional<at::ScalarType> out);

Pair conv_fwd(const Tensor& x, const Tensor& weight, const Tensor& bias, const Tensor& residual, const Tensor& init, bool want_final, bool silu,
              const Tensor& cu, int64_t head_num);
std::vector<Tensor> conv_bwd(const Tensor& x, const Tensor& weight, const Tensor& dy, const Tensor& bias, const Tensor& init, const Tensor& dht,
                             bool silu, const Tensor& cu, const Tensor& y_pre, bool want_dh0, at::ScalarType dw_dtype, at::ScalarType db_dtype);
Pair conv(const Tensor& x, const Tensor& weight, const Tensor& bias, const Tensor& residual, const Tensor& init, bool want_final, bool silu,
          const Tensor& cu);
Tensor conv_update(const Tensor& x, const Tensor& cache, const Tensor& residual, const Tensor& weight, const Tensor& bias, bool silu,
                   const Tensor& cache_indices, const Tensor& accepted, int64_t pad_slot);

Pair recurrent_fused(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale, const Tensor& h0,
                     bool want_final, bool l2norm, const Tensor& cu, bool v_first, bool inplace, const Tensor& gk);
Tensor recurrent_pool(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& state, const Tensor& beta, double scale,
                      const Tensor& lengths, const Tensor& indices, const Tensor& accepted, const Tensor& g);
Pair recurrent_kda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& h0, const Tensor& cu,
                   const Tensor& indices, const Tensor& a_log, const Tensor& dt_bias, const Tensor& accepted, double scale, bool inplace,
                   bool l2norm, int64_t gate_mode, int64_t beta_mode, double lower_bound, bool v_first, int64_t seq_num);

// What the GDN forward leaves for its backward.  The operators keep all of it in one allocation (`slab`): a dozen small tensors cost the
// host more than the launches of a short prompt.  Callers that want the tensors themselves get them one by one.
struct GdnSaved {
  enum Piece { kGam, kX, kS, kVn, kP, kSegM, kQn, kKn, kQr, kKr, kPieces };      // kSegM: transition matrices of split chains
  Tensor slab, piece[kPieces];
  std::array<int64_t, kPieces> at{};      // byte offsets in the slab, -1: absent
  int64_t hk = 0;                         // q/k heads
  Geometry geo;
};
std::tuple<Tensor, Tensor, GdnSaved> gdn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale,
                                             const Tensor& h0, bool want_final, const Tensor& cu, bool save, std::optional<at::ScalarType> out, bool l2norm,
                                             bool slab);
struct GradTypes {
  at::ScalarType q, k, v, g, beta;
};
std::vector<Tensor> gdn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const GdnSaved& saved, const Tensor& d_o,
                            const Tensor& dht, double scale, bool want_dh0, GradTypes types);
Pair gdn(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale, const Tensor& h0, bool want_final,
         const Tensor& cu, std::optional<at::ScalarType> out, bool l2norm);

struct KdaOptions {
  double scale = 1.0, lower_bound = 0.0;
  int64_t gate_mode = 0;
  bool want_final = false, l2norm = false, keep = false, want_gk = false;
  std::optional<at::ScalarType> out;
};
struct KdaResult {
  Tensor o, ht, gk, saved, q_rstd, k_rstd;
};
KdaResult kda_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& h0, const Tensor& a_log,
                  const Tensor& dt_bias, const Geometry& geo, const KdaOptions& o, const Tensor& aqk, const Tensor& akk);
std::vector<Tensor> kda_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale, const Tensor& h0,
                            const Tensor& d_o, const Tensor& dht, const Geometry& geo, GradTypes types, const Tensor& saved,
                            const Tensor& q_rstd = Tensor(), const Tensor& k_rstd = Tensor());
struct KdaCall {
  KdaResult r;
  Geometry geo;
  Tensor q, k, v, beta;      // the row-major inputs, when the saved images are returned
};
// The operator: differentiable in q, k, v, g, beta and h0 when the gate is given activated (gate_mode 0).
KdaCall kda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& h0, const Tensor& a_log,
            const Tensor& dt_bias, const Tensor& cu, KdaOptions o, const Tensor& aqk, const Tensor& akk, bool return_saved);
// Views of a head-first batch as one sequence of B*H heads; undefined tensors when it cannot or need not be folded.
Tensor fold(const Tensor& t);
std::array<Tensor, 3> fold_plan(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu);

}  // namespace fla_host
