#include "runtime.h"
#include <ATen/cuda/CUDAContext.h>
#include <Python.h>
#include <c10/cuda/CUDAException.h>
#include <vector>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

namespace fla_host {

Library lib;
bool check_status = false;

static const char* status_name(int s) {
  switch (s) {
    case FLA_ERR_NULL: return "FLA_ERR_NULL (required tensor missing)";
    case FLA_ERR_SHAPE: return "FLA_ERR_SHAPE (unsupported or inconsistent shape)";
    case FLA_ERR_DTYPE: return "FLA_ERR_DTYPE (unsupported dtype)";
    case FLA_ERR_LAYOUT: return "FLA_ERR_LAYOUT (stride / alignment requirement not met)";
    case FLA_ERR_WORKSPACE: return "FLA_ERR_WORKSPACE (workspace too small)";
    case FLA_ERR_CUDA: return "FLA_ERR_CUDA (CUDA runtime error)";
    case FLA_ERR_VALUE: return "FLA_ERR_VALUE (scalar argument out of range)";
    case FLA_ERR_TIMEOUT: return "FLA_ERR_TIMEOUT (device-side wait ran out)";
    case FLA_ERR_TOO_LARGE: return "FLA_ERR_TOO_LARGE (problem exceeds the built-in scratch of an allocation-free entry point)";
  }
  return "?";
}
void fail(const char* op, int status) { TORCH_CHECK(false, op, " failed with status=", status, ": ", status_name(status)); }

int32_t dtype_code(at::ScalarType t, const char* name) {
  switch (t) {
    case at::kFloat: return FLA_F32;
    case at::kBFloat16: return FLA_BF16;
    case at::kHalf: return FLA_F16;
    case at::kInt: return FLA_I32;
    case at::kLong: return FLA_I64;
    default: TORCH_CHECK_TYPE(false, name, ": unsupported dtype ", t);
  }
}

at::Device Device::get() const {
  TORCH_CHECK(set_, op_, ": no tensors given");
  static bool checked[64] = {};
  const int i = dev_.index();
  if (i >= 64 || !checked[i]) {
    const auto* prop = at::cuda::getDeviceProperties(i);
    TORCH_CHECK(prop->major == 10, op_, ": libfla_b200 is built for sm_100a only; device ", dev_, " is sm_", prop->major, "x");
    if (i < 64) checked[i] = true;
  }
  return dev_;
}

// The checked mode reads the word through the Python layer, where callers that watch or replace the reader expect it.
void raise_device_status(const char* op, const Tensor& ws) {
  const PyGILState_STATE gil = PyGILState_Ensure();
  PyObject* mod = PyImport_ImportModule("fla_b200._runtime");
  PyObject* w = mod ? THPVariable_Wrap(ws) : nullptr;
  PyObject* r = w ? PyObject_CallMethod(mod, "read_device_status", "Os", w, op) : nullptr;
  Py_XDECREF(w);
  Py_XDECREF(mod);
  if (!r) {
    python_error err;
    err.persist();
    PyGILState_Release(gil);
    throw std::move(err);
  }
  Py_DECREF(r);
  PyGILState_Release(gil);
}

Tensor convert(const Tensor& t, at::ScalarType dtype, const char* op) {
  TORCH_CHECK(t.dim() >= 1 && t.dim() <= 4, op, ": conversion takes 1 to 4 dims, got ", t.dim());
  const at::Device d = Device(op)(t).get();
  Tensor out = empty(t.sizes(), dtype, d);
  if (!t.numel()) return out;
  const Tensor src = (t.size(-1) != 1 && t.stride(-1) != 1) ? t.contiguous() : t;
  const fla_tensor_t s = desc(src), o = desc(out);
  one_phase(op, d, lib.convert, &s, &o);
  return out;
}

struct ConvertFn : torch::autograd::Function<ConvertFn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& t, int64_t dtype, const char* op) {
    ctx->saved_data["dtype"] = int64_t(t.scalar_type());
    return convert(t, at::ScalarType(dtype), op);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grad) {
    return {convert(grad[0], at::ScalarType(ctx->saved_data["dtype"].toInt()), "convert"), Tensor(), Tensor()};
  }
};
Tensor to_dtype(const Tensor& t, at::ScalarType dtype, const char* op) {
  if (!t.defined() || t.scalar_type() == dtype) return t;
  if (!t.requires_grad() || !at::GradMode::is_enabled()) return convert(t, dtype, op);
  return ConvertFn::apply(t, int64_t(dtype), op);
}

// Boundaries that are on the device, read back by the kernel that makes the chunk offsets: it writes them into pinned memory, where this
// thread polls for the tag of the call.  A copy into pageable memory and the offsets' launch behind it took 12 us more per packed call, all of
// it with an idle device.  False where the plain copy has to do (a captured stream, whose copy reports the error; very many sequences).
static bool read_bounds(const char* op, const Tensor& cu, const Tensor& co, at::Device d, std::vector<int32_t>& out) {
  struct Pinned {
    int32_t* p = nullptr;
    int32_t tag = 0;
  };
  constexpr int64_t kMost = 4095;
  thread_local Pinned pin;      // (lives as long as the process: CUDA may be gone when a thread ends)
  const int64_t n = cu.numel();
  if (n < 2 || n > kMost) return false;
  c10::cuda::CUDAGuard guard(d);
  const cudaStream_t stream = static_cast<cudaStream_t>(current_stream(d));
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return false;
  if (!pin.p) {
    if (cudaHostAlloc(reinterpret_cast<void**>(&pin.p), (kMost + 1) * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      pin.p = nullptr;
      return false;
    }
    pin.p[0] = 0;
  }
  pin.tag = pin.tag == 0x7fffffff ? 1 : pin.tag + 1;
  const fla_tensor_t a = desc(cu), b = desc(co);
  ok_or_throw(op, lib.chunk_bounds(&a, &b, pin.p, pin.tag, stream));
  for (uint32_t spin = 0; __atomic_load_n(pin.p, __ATOMIC_ACQUIRE) != pin.tag; ++spin) {
    if ((spin & 0xfff) != 0xfff) continue;
    const cudaError_t e = cudaStreamQuery(stream);
    if (e == cudaErrorNotReady) continue;
    C10_CUDA_CHECK(e);
    TORCH_CHECK(__atomic_load_n(pin.p, __ATOMIC_ACQUIRE) == pin.tag, op, ": the sequence boundaries did not arrive");
  }
  out.assign(pin.p + 1, pin.p + 1 + n);
  return true;
}

// Packed batches: the kernels' grids and the sizes of the saved tensors follow from the lengths, so the boundaries have to be
// known on the host.  A device tensor is read back once (its stream is waited for); the chunk offsets are made on the
// device from the boundaries that are already there.
Geometry geometry(const char* op, int64_t B, int64_t T, const Tensor& cu_seqlens, at::Device d) {
  Geometry geo;
  if (!cu_seqlens.defined()) {
    geo.N = B;
    geo.max_len = T;
    geo.chunks = B * ((T + kChunk - 1) / kChunk);
    return geo;
  }
  TORCH_CHECK(B == 1, op, ": cu_seqlens requires batch size 1 (packed sequences)");
  Tensor host;
  std::vector<int32_t> bounds;
  if (cu_seqlens.device() == d && cu_seqlens.dim() == 1) {
    geo.cu = cu_seqlens.to(at::kInt).contiguous();
    geo.co = empty({cu_seqlens.numel()}, at::kInt, d);
  }
  {
    PyThreadState* ts = PyGILState_Check() ? PyEval_SaveThread() : nullptr;
    try {
      if (!geo.co.defined() || !read_bounds(op, geo.cu, geo.co, d, bounds)) host = cu_seqlens.to(at::kCPU, at::kInt).contiguous();
    } catch (...) {
      if (ts) PyEval_RestoreThread(ts);
      throw;
    }
    if (ts) PyEval_RestoreThread(ts);
  }
  const int32_t* cu = host.defined() ? host.data_ptr<int32_t>() : bounds.data();
  const int64_t n = host.defined() ? host.numel() : int64_t(bounds.size());
  bool fine = n >= 2 && cu[0] == 0;
  for (int64_t i = 0; fine && i + 1 < n; ++i) fine = cu[i + 1] >= cu[i];
  TORCH_CHECK(fine, "cu_seqlens must start at 0 and be non-decreasing, got ", std::vector<int64_t>(cu, cu + n));
  geo.N = n - 1;
  for (int64_t i = 0; i < geo.N; ++i) {
    const int64_t len = cu[i + 1] - cu[i];
    geo.max_len = std::max(geo.max_len, len);
    geo.chunks += (len + kChunk - 1) / kChunk;
  }
  TORCH_CHECK(cu[n - 1] == T, op, ": cu_seqlens[-1]=", cu[n - 1], " must equal T=", T);
  if (!host.defined()) return geo;
  if (!geo.co.defined()) {
    geo.cu = host.to(d);
    geo.co = empty({n}, at::kInt, d);
  }
  const fla_tensor_t a = desc(geo.cu), b = desc(geo.co);
  one_phase(op, d, lib.chunk_offsets, &a, &b);
  return geo;
}

Pair l2norm_fwd(const Tensor& x, double eps, std::optional<at::ScalarType> out) {
  const at::Device d = Device("l2norm_fwd")(x).get();
  Tensor x2 = x.reshape({-1, x.size(-1)});
  if (x2.stride(-1) != 1) x2 = x2.contiguous();
  Tensor y = empty(x2.sizes(), out.value_or(x.scalar_type()), d), rstd = empty({x2.size(0)}, at::kFloat, d);
  fla_l2norm_args a{};
  a.x = desc(x2), a.y = desc(y), a.rstd = desc(rstd), a.eps = float(eps);
  one_phase("l2norm_fwd", d, lib.l2norm_fwd, &a);
  return {y.view(x.sizes()), rstd.view(x.sizes().slice(0, x.dim() - 1))};
}
Tensor l2norm_bwd(const Tensor& y, const Tensor& rstd, const Tensor& dy, double eps, std::optional<at::ScalarType> out) {
  const at::Device d = Device("l2norm_bwd")(y)(rstd)(dy).get();
  auto rows = [](const Tensor& t) {
    Tensor r = t.reshape({-1, t.size(-1)});
    return r.stride(-1) == 1 ? r : r.contiguous();
  };
  const Tensor y2 = rows(y), dy2 = rows(dy), r = rstd.reshape(-1).contiguous();
  Tensor dx = empty(y2.sizes(), out.value_or(y.scalar_type()), d);
  fla_l2norm_args a{};
  a.y = desc(y2), a.rstd = desc(r), a.dy = desc(dy2), a.dx = desc(dx), a.eps = float(eps);
  one_phase("l2norm_bwd", d, lib.l2norm_bwd, &a);
  return dx.view(y.sizes());
}

}  // namespace fla_host
