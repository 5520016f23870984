// The Python face of the binding: plain positional C functions.  Signatures, defaults and documentation live in
// fla_b200/ops/*.py, whose functions end in one call of these.
#include <Python.h>
#include <dlfcn.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include "runtime.h"

namespace fla_host {
namespace {

// Positional arguments of one call, taken in order.
class Args {
 public:
  Args(PyObject* const* a, Py_ssize_t n, Py_ssize_t want) : a_(a) {
    TORCH_CHECK_TYPE(n == want, "fla_b200 binding: expected ", want, " arguments, got ", n);
  }
  Tensor tensor() {
    PyObject* o = a_[i_++];
    if (o == Py_None) return Tensor();
    TORCH_CHECK_TYPE(THPVariable_Check(o), "argument ", i_, " must be a torch.Tensor or None, got ", Py_TYPE(o)->tp_name);
    return THPVariable_Unpack(o);
  }
  double number() {
    const double x = PyFloat_AsDouble(a_[i_++]);
    if (x == -1.0 && PyErr_Occurred()) throw python_error();
    return x;
  }
  int64_t integer() {
    const long long x = PyLong_AsLongLong(a_[i_++]);
    if (x == -1 && PyErr_Occurred()) throw python_error();
    return x;
  }
  bool flag() {
    const int x = PyObject_IsTrue(a_[i_++]);
    if (x < 0) throw python_error();
    return x != 0;
  }
  std::optional<at::ScalarType> dtype() {
    PyObject* o = a_[i_++];
    if (o == Py_None) return std::nullopt;
    TORCH_CHECK_TYPE(THPDtype_Check(o), "argument ", i_, " must be a torch.dtype or None");
    return reinterpret_cast<THPDtype*>(o)->scalar_type;
  }
  at::ScalarType dtype_or(at::ScalarType other) { return dtype().value_or(other); }
  // a tensor, or the same integers as a Python sequence
  Tensor boundaries() {
    PyObject* o = a_[i_];
    if (o == Py_None || THPVariable_Check(o)) return tensor();
    ++i_;
    PyObject* seq = PySequence_Fast(o, "cu_seqlens must be a tensor or a sequence of integers");
    if (!seq) throw python_error();
    Tensor t = at::empty({PySequence_Fast_GET_SIZE(seq)}, at::kInt);
    int32_t* p = t.data_ptr<int32_t>();
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) p[i] = int32_t(PyLong_AsLong(PySequence_Fast_GET_ITEM(seq, i)));
    Py_DECREF(seq);
    if (PyErr_Occurred()) throw python_error();
    return t;
  }

 private:
  PyObject* const* a_;
  Py_ssize_t i_ = 0;
};

PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* pack(std::initializer_list<PyObject*> items) {
  PyObject* r = PyTuple_New(Py_ssize_t(items.size()));
  Py_ssize_t i = 0;
  for (PyObject* o : items) PyTuple_SET_ITEM(r, i++, o);
  return r;
}
PyObject* pack(const Pair& p) { return pack({wrap(p.first), wrap(p.second)}); }
PyObject* pack(const std::vector<Tensor>& v) {
  PyObject* r = PyTuple_New(Py_ssize_t(v.size()));
  for (size_t i = 0; i < v.size(); ++i) PyTuple_SET_ITEM(r, Py_ssize_t(i), wrap(v[i]));
  return r;
}

#define FLA_PY(name, nargs)                                                             \
  PyObject* name##_body(Args& a);                                                       \
  PyObject* name(PyObject*, PyObject* const* argv, Py_ssize_t n) {                      \
    HANDLE_TH_ERRORS                                                                    \
    Args a(argv, n, nargs);                                                             \
    return name##_body(a);                                                              \
    END_HANDLE_TH_ERRORS                                                                \
  }                                                                                     \
  PyObject* name##_body(Args& a)

FLA_PY(py_bind, 1) {      // the dlopen handle of libfla_b200.so
  void* h = reinterpret_cast<void*>(a.integer());
#define FLA_LOOK(n)                                                                                  \
  lib.n = reinterpret_cast<decltype(lib.n)>(dlsym(h, "fla_b200_" #n));                               \
  TORCH_CHECK(lib.n, "libfla_b200.so does not export fla_b200_" #n);
  FLA_HOST_FNS(FLA_LOOK)
#undef FLA_LOOK
  Py_RETURN_NONE;
}
FLA_PY(py_check_status, 1) {
  check_status = a.flag();
  Py_RETURN_NONE;
}
FLA_PY(py_convert, 2) {
  const Tensor t = a.tensor();
  const auto dt = a.dtype();
  TORCH_CHECK(t.defined() && dt, "convert: a tensor and a dtype are needed");
  return wrap(convert(t, *dt, "convert"));
}
FLA_PY(py_to_dtype, 2) {
  const Tensor t = a.tensor();
  const auto dt = a.dtype();
  TORCH_CHECK(dt, "to_dtype: a dtype is needed");
  return wrap(to_dtype(t, *dt, "convert"));
}
FLA_PY(py_l2norm_fwd, 3) {
  const Tensor x = a.tensor();
  const double eps = a.number();
  return pack(l2norm_fwd(x, eps, a.dtype()));
}
FLA_PY(py_l2norm_bwd, 4) {
  const Tensor y = a.tensor(), rstd = a.tensor(), dy = a.tensor();
  return wrap(l2norm_bwd(y, rstd, dy, a.number(), std::nullopt));
}
FLA_PY(py_conv, 8) {
  const Tensor x = a.tensor(), w = a.tensor(), b = a.tensor(), r = a.tensor(), init = a.tensor();
  const bool fin = a.flag(), silu = a.flag();
  return pack(conv(x, w, b, r, init, fin, silu, a.tensor()));
}
FLA_PY(py_conv_fwd, 9) {
  const Tensor x = a.tensor(), w = a.tensor(), b = a.tensor(), r = a.tensor(), init = a.tensor();
  const bool fin = a.flag(), silu = a.flag();
  const Tensor cu = a.tensor();
  return pack(conv_fwd(x, w, b, r, init, fin, silu, cu, a.integer()));
}
FLA_PY(py_conv_bwd, 10) {
  const Tensor x = a.tensor(), w = a.tensor(), dy = a.tensor(), b = a.tensor(), init = a.tensor(), dht = a.tensor();
  const bool silu = a.flag();
  const Tensor cu = a.tensor(), ypre = a.tensor();
  return pack(conv_bwd(x, w, dy, b, init, dht, silu, cu, ypre, a.flag(), at::kFloat, at::kFloat));
}
FLA_PY(py_conv_update, 9) {
  const Tensor x = a.tensor(), cache = a.tensor(), r = a.tensor(), w = a.tensor(), b = a.tensor();
  const bool silu = a.flag();
  const Tensor idx = a.tensor(), acc = a.tensor();
  return wrap(conv_update(x, cache, r, w, b, silu, idx, acc, a.integer()));
}
FLA_PY(py_recurrent_fused, 13) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor();
  const double scale = a.number();
  const Tensor h0 = a.tensor();
  const bool fin = a.flag(), l2 = a.flag();
  const Tensor cu = a.boundaries();
  const bool vf = a.flag(), inplace = a.flag();
  return pack(recurrent_fused(q, k, v, g, beta, scale, h0, fin, l2, cu, vf, inplace, a.tensor()));
}
FLA_PY(py_recurrent_pool, 10) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), state = a.tensor(), beta = a.tensor();
  const double scale = a.number();
  const Tensor len = a.tensor(), idx = a.tensor(), acc = a.tensor();
  return wrap(recurrent_pool(q, k, v, state, beta, scale, len, idx, acc, a.tensor()));
}
FLA_PY(py_recurrent_kda, 19) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor(), h0 = a.tensor(), cu = a.tensor(), idx = a.tensor(),
               al = a.tensor(), db = a.tensor(), acc = a.tensor();
  const double scale = a.number();
  const bool inplace = a.flag(), l2 = a.flag();
  const int64_t gm = a.integer(), bm = a.integer();
  const double lower = a.number();
  const bool vf = a.flag();
  return pack(recurrent_kda(q, k, v, g, beta, h0, cu, idx, al, db, acc, scale, inplace, l2, gm, bm, lower, vf, a.integer()));
}
PyObject* geometry_items(const Geometry& g) {      // (cu, co, N, max_len, total_chunks)
  return pack({wrap(g.cu), wrap(g.co), PyLong_FromLongLong(g.N), PyLong_FromLongLong(g.max_len), PyLong_FromLongLong(g.chunks)});
}
Geometry geometry_of(Args& a) {
  Geometry g;
  g.cu = a.tensor(), g.co = a.tensor();
  g.N = a.integer(), g.max_len = a.integer(), g.chunks = a.integer();
  return g;
}
FLA_PY(py_geometry, 4) {
  const int64_t B = a.integer(), T = a.integer();
  const Tensor cu = a.boundaries(), on = a.tensor();
  return geometry_items(geometry("cu_seqlens", B, T, cu, on.device()));
}
FLA_PY(py_gdn, 11) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor();
  const double scale = a.number();
  const Tensor h0 = a.tensor();
  const bool fin = a.flag();
  const Tensor cu = a.boundaries();
  const auto out = a.dtype();
  return pack(gdn(q, k, v, g, beta, scale, h0, fin, cu, out, a.flag()));
}
FLA_PY(py_gdn_fwd, 11) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor();
  const double scale = a.number();
  const Tensor h0 = a.tensor();
  const bool fin = a.flag();
  const Tensor cu = a.boundaries();
  const bool save = a.flag();
  auto [o, ht, s] = gdn_fwd(q, k, v, g, beta, scale, h0, fin, cu, save, a.dtype(), false, false);
  const Tensor* t = s.piece;
  return pack({wrap(o), wrap(ht), wrap(t[GdnSaved::kGam]), wrap(t[GdnSaved::kX]), wrap(t[GdnSaved::kS]), wrap(t[GdnSaved::kVn]), wrap(t[GdnSaved::kP]),
               wrap(t[GdnSaved::kSegM]), geometry_items(s.geo)});
}
FLA_PY(py_gdn_bwd, 24) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), beta = a.tensor();
  GdnSaved s;
  for (int i = GdnSaved::kGam; i <= GdnSaved::kSegM; ++i) s.piece[i] = a.tensor();
  s.at.fill(-1);
  s.geo = geometry_of(a);
  const Tensor d_o = a.tensor(), dht = a.tensor();
  const double scale = a.number();
  const bool dh0 = a.flag();
  GradTypes t;
  t.q = a.dtype_or(at::kBFloat16), t.k = a.dtype_or(at::kBFloat16), t.v = a.dtype_or(at::kBFloat16), t.g = a.dtype_or(at::kBFloat16);
  t.beta = a.dtype_or(at::kBFloat16);
  return pack(gdn_bwd(q, k, v, beta, s, d_o, dht, scale, dh0, t));
}
FLA_PY(py_kda_fwd, 22) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor(), h0 = a.tensor(), al = a.tensor(), db = a.tensor();
  const Geometry geo = geometry_of(a);
  KdaOptions o;
  o.scale = a.number(), o.lower_bound = a.number(), o.gate_mode = a.integer();
  o.want_final = a.flag(), o.keep = a.flag(), o.want_gk = a.flag();
  o.out = a.dtype();
  const Tensor aqk = a.tensor(), akk = a.tensor();
  const KdaResult r = kda_fwd(q, k, v, g, beta, h0, al, db, geo, o, aqk, akk);
  return pack({wrap(r.o), wrap(r.ht), wrap(r.gk), wrap(r.saved)});
}
FLA_PY(py_kda_bwd, 20) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor();
  const double scale = a.number();
  const Tensor h0 = a.tensor(), d_o = a.tensor(), dht = a.tensor();
  const Geometry geo = geometry_of(a);
  GradTypes t;
  t.q = a.dtype_or(at::kFloat), t.k = a.dtype_or(at::kFloat), t.v = a.dtype_or(at::kFloat), t.g = a.dtype_or(at::kFloat), t.beta = a.dtype_or(at::kFloat);
  return pack(kda_bwd(q, k, v, g, beta, scale, h0, d_o, dht, geo, t, a.tensor()));
}
FLA_PY(py_kda, 19) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor(), h0 = a.tensor(), al = a.tensor(), db = a.tensor(),
               cu = a.boundaries();
  KdaOptions o;
  o.scale = a.number(), o.lower_bound = a.number(), o.gate_mode = a.integer();
  o.want_final = a.flag(), o.l2norm = a.flag(), o.keep = a.flag(), o.want_gk = a.flag();
  o.out = a.dtype();
  const Tensor aqk = a.tensor(), akk = a.tensor();
  const KdaCall c = kda(q, k, v, g, beta, h0, al, db, cu, o, aqk, akk, false);
  if (o.want_gk) return pack({wrap(c.r.o), wrap(c.r.ht), wrap(c.r.gk)});
  return pack({wrap(c.r.o), wrap(c.r.ht)});
}
// The forward with its operand images kept: (o, ht, saved, geometry, (q, k, v, beta) as the kernels read them).
FLA_PY(py_kda_saved, 13) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), g = a.tensor(), beta = a.tensor(), h0 = a.tensor(), cu = a.boundaries();
  KdaOptions o;
  o.scale = a.number(), o.want_final = a.flag(), o.l2norm = a.flag();
  o.out = a.dtype();
  const Tensor aqk = a.tensor(), akk = a.tensor();
  const KdaCall c = kda(q, k, v, g, beta, h0, Tensor(), Tensor(), cu, o, aqk, akk, true);
  return pack({wrap(c.r.o), wrap(c.r.ht), wrap(c.r.saved), geometry_items(c.geo), pack({wrap(c.q), wrap(c.k), wrap(c.v), wrap(c.beta)})});
}
FLA_PY(py_fold, 1) { return wrap(fold(a.tensor())); }
FLA_PY(py_fold_plan, 4) {
  const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor();
  const auto f = fold_plan(q, k, v, a.boundaries());
  if (!f[0].defined()) Py_RETURN_NONE;
  return pack({wrap(f[0]), wrap(f[1]), wrap(f[2])});
}

#define FLA_M(py, fn) {py, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FLA_M("bind", py_bind), FLA_M("check_status", py_check_status), FLA_M("convert", py_convert), FLA_M("to_dtype", py_to_dtype),
    FLA_M("l2norm_fwd", py_l2norm_fwd), FLA_M("l2norm_bwd", py_l2norm_bwd), FLA_M("conv", py_conv), FLA_M("conv_fwd", py_conv_fwd),
    FLA_M("conv_bwd", py_conv_bwd), FLA_M("conv_update", py_conv_update), FLA_M("recurrent_fused", py_recurrent_fused),
    FLA_M("recurrent_pool", py_recurrent_pool), FLA_M("recurrent_kda", py_recurrent_kda), FLA_M("geometry", py_geometry), FLA_M("gdn", py_gdn),
    FLA_M("gdn_fwd", py_gdn_fwd), FLA_M("gdn_bwd", py_gdn_bwd), FLA_M("kda_fwd", py_kda_fwd), FLA_M("kda_bwd", py_kda_bwd),
    FLA_M("kda", py_kda), FLA_M("kda_saved", py_kda_saved),
    FLA_M("fold", py_fold), FLA_M("fold_plan", py_fold_plan), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "PyTorch binding of libfla_b200.so", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace fla_host

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host() { return PyModule_Create(&fla_host::module_def); }
