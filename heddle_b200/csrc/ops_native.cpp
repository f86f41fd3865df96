// Host path of the tensor-level calls of heddle_b200/ops.py: reads shapes, strides and pointers from the tensors, allocates the
// results, fills the C ABI's argument structs and calls the library, as ops.py does it in Python.
//
// Where a call's kernels take a few microseconds its time is the host's: in Python the wrappers cost 8 to 15 us a call (34 for a
// backward pass), about 3 us of which are launches.  Only plain calls are taken here: exact torch.Tensor objects, dense, on the
// current device, with shapes, types and strides the kernels read in place, no mode or transform in force.  Everything else gets
// NotImplemented, and ops.py goes on with its general path, which converts, copies or refuses as ever.  Nothing is kept from one
// call for the next.  us of host time a call, in Python -> here:
// attention 12.0 -> 6.7, with few query rows 13.6 -> 6.5, backward 34 -> 16, H2O score 19.8 -> 9.1, GEMM 10.0 -> 4.6, batched 13.0 -> 4.4,
// RMS statistic 8.1 -> 3.7, softmax 9.1 -> 3.8, rowwise program 13.5 -> 4.3; a compiled decoder layer of 1024 hidden, 25 rows 188 -> 98.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <string>

#include "../../include/heddle_b200.h"

namespace {

// entry points of the library that ops.py has loaded, bound once
struct Lib {
  decltype(&hb_fa_fwd) fa_fwd;
  decltype(&hb_fa_fwd_workspace) fa_fwd_workspace;
  decltype(&hb_fa_fwd_ws) fa_fwd_ws;
  decltype(&hb_fa_bwd_dkdv_workspace) fa_bwd_dkdv_workspace;
  decltype(&hb_fa_bwd) fa_bwd;
  decltype(&hb_h2o_score) h2o_score;
  decltype(&hb_gemm_epilogue) gemm_epilogue;
  decltype(&hb_rms_rowstat) rms_rowstat;
  decltype(&hb_row_softmax) row_softmax;
  decltype(&hb_rowwise_program) rowwise_program;
} lib;
PyObject* g_check = nullptr;    // _lib.check: raises for a status
PyObject* g_ew_ops = nullptr;   // _lib.EW_OPS, _lib.EW_SRCS
PyObject* g_ew_srcs = nullptr;

PyObject* general() { Py_RETURN_NOTIMPLEMENTED; }

// Calls the library without the interpreter lock, as a foreign call from Python does.
template <typename F>
int unlocked(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS rc = f();
  Py_END_ALLOW_THREADS return rc;
}

PyObject* raise_status(int rc) {
  PyObject* r = PyObject_CallFunction(g_check, "i", rc);
  if (r == nullptr) return nullptr;
  Py_DECREF(r);
  PyErr_SetString(PyExc_RuntimeError, "heddle_b200: a failed call raised nothing");
  return nullptr;
}

const c10::DispatchKeySet& special_keys() {
  using K = c10::DispatchKey;
  static const c10::DispatchKeySet keys({K::Python, K::PythonTLSSnapshot, K::FuncTorchBatched, K::FuncTorchGradWrapper,
                                         K::FuncTorchVmapMode, K::FuncTorchDynamicLayerFrontMode, K::FuncTorchDynamicLayerBackMode,
                                         K::Functionalize, K::Conjugate, K::Negative, K::ZeroTensor, K::Batched,
                                         K::BatchedNestedTensor, K::VmapMode, K::Tracer, K::DeferredInit, K::TESTING_ONLY_GenericMode});
  return keys;
}

// No mode or transform in force that would want to see the calls the general path makes.
bool plain_context() {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled()) return false;
  return !c10::impl::tls_local_dispatch_key_set().included_.has_any(special_keys());
}

// The tensor behind an exact torch.Tensor (or Parameter) that is dense, not empty and on the device `index` (any where it is -1).
const at::Tensor* plain(PyObject* o, int index) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.key_set().has_any(special_keys()) || t.numel() == 0) return nullptr;
  if (index >= 0 && t.device().index() != index) return nullptr;
  return &t;
}

// The same on the current device, whose index is returned too.
const at::Tensor* plain_first(PyObject* o, int& index) {
  const at::Tensor* t = plain(o, -1);
  if (t == nullptr) return nullptr;
  index = t->device().index();
  return index == c10::cuda::current_device() ? t : nullptr;
}

int dtype16(const at::Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? HB_BF16 : t.scalar_type() == at::kHalf ? HB_FP16 : -1;
}

void* stream_of(int index) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(index)).stream(); }
at::Tensor empty_like_options(const at::Tensor& t, at::IntArrayRef sizes, at::ScalarType type) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(t.device()));
}
bool aligned16(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }
bool fits_int(int64_t v) { return v >= 0 && v <= std::numeric_limits<int32_t>::max(); }
bool contiguous_fp32(const at::Tensor& t, int64_t n) { return t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() == n; }

// A Python number as double; false (no error set) for anything else.
bool number(PyObject* o, double& v) {
  v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool integer(PyObject* o, int64_t& v) {
  if (!PyLong_CheckExact(o)) return false;
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// 0 "bhsd", 1 "bshd", -1 anything else
int layout_of(PyObject* o) {
  if (!PyUnicode_CheckExact(o)) return -1;
  if (PyUnicode_CompareWithASCIIString(o, "bhsd") == 0) return 0;
  return PyUnicode_CompareWithASCIIString(o, "bshd") == 0 ? 1 : -1;
}

struct Dims {
  int64_t B, Hq, Hkv, Sq, Skv, D;
  int h, s;  // axes of heads and positions
};
// Extents of q [.., D] and k of the same layout; false where the general path has something to say.
bool attention_dims(const at::Tensor& q, const at::Tensor& k, int layout, Dims& d) {
  if (layout < 0 || q.dim() != 4 || k.dim() != 4 || q.stride(3) != 1 || k.stride(3) != 1 || k.scalar_type() != q.scalar_type()) return false;
  d.h = layout == 0 ? 1 : 2;
  d.s = layout == 0 ? 2 : 1;
  d.B = q.size(0);
  d.Hq = q.size(d.h);
  d.Sq = q.size(d.s);
  d.D = q.size(3);
  d.Hkv = k.size(d.h);
  d.Skv = k.size(d.s);
  return k.size(0) == d.B && k.size(3) == d.D && fits_int(d.B) && fits_int(d.Hq) && fits_int(d.Sq) && fits_int(d.Skv) && fits_int(d.Hkv) && fits_int(d.D);
}
template <typename Args>
void fill_dims(Args& a, const Dims& d, bool causal, double scale, int dtype, int device) {
  a.B = static_cast<int32_t>(d.B);
  a.Hq = static_cast<int32_t>(d.Hq);
  a.Hkv = static_cast<int32_t>(d.Hkv);
  a.Sq = static_cast<int32_t>(d.Sq);
  a.Skv = static_cast<int32_t>(d.Skv);
  a.D = static_cast<int32_t>(d.D);
  a.causal = causal ? 1 : 0;
  a.softmax_scale = static_cast<float>(scale);
  a.dtype = dtype;
  a.stream = stream_of(device);
}
bool softmax_scale(PyObject* o, int64_t D, double& scale) {
  if (o == Py_None) {
    scale = 1.0 / std::sqrt(static_cast<double>(D));
    return true;
  }
  return number(o, scale);
}

// fa_fwd(q, k, v, causal, softmax_scale, layout, return_lse, out, scales, bshd_out): `out` None or a tensor; bshd_out: a new
// result of layout "bhsd" is stored as [B, S, H, D]
PyObject* fa_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 10 || !plain_context()) return general();
  int dev;
  const at::Tensor* q = plain_first(args[0], dev);
  if (q == nullptr) return general();
  const at::Tensor *k = plain(args[1], dev), *v = plain(args[2], dev);
  if (k == nullptr || v == nullptr) return general();
  const int layout = layout_of(args[5]);
  const bool fp8 = q->scalar_type() == at::kFloat8_e4m3fn;
  const int dtype = fp8 ? HB_FP8_E4M3 : dtype16(*q);
  Dims d;
  double scale;
  if (dtype < 0 || !attention_dims(*q, *k, layout, d) || v->sizes() != k->sizes() || v->stride(3) != 1 || v->scalar_type() != q->scalar_type() ||
      !softmax_scale(args[4], d.D, scale))
    return general();
  const int causal = PyObject_IsTrue(args[3]), want_lse = PyObject_IsTrue(args[6]), bshd_out = PyObject_IsTrue(args[9]);
  if (causal < 0 || want_lse < 0 || bshd_out < 0) return nullptr;
  hb_fa_args a;
  std::memset(&a, 0, sizeof(a));
  if (args[8] != Py_None) {
    double s[3];
    if (!PyTuple_CheckExact(args[8]) || PyTuple_GET_SIZE(args[8]) != 3) return general();
    for (int i = 0; i < 3; ++i)
      if (!number(PyTuple_GET_ITEM(args[8], i), s[i])) return general();
    a.q_scale = static_cast<float>(s[0]);
    a.k_scale = static_cast<float>(s[1]);
    a.v_scale = static_cast<float>(s[2]);
  }
  const at::ScalarType out_type = fp8 ? at::kBFloat16 : q->scalar_type();
  at::Tensor o;
  if (args[7] != Py_None) {
    const at::Tensor* given = plain(args[7], dev);
    if (given == nullptr || given->sizes() != q->sizes() || given->scalar_type() != out_type || given->stride(3) != 1) return general();
    o = *given;
  } else if (bshd_out && layout == 0) {
    o = empty_like_options(*q, {d.B, d.Sq, d.Hq, d.D}, out_type).transpose(1, 2);
  } else {
    o = empty_like_options(*q, q->sizes(), out_type);
  }
  at::Tensor lse;
  if (want_lse) lse = empty_like_options(*q, {d.B, d.Hq, d.Sq}, at::kFloat);
  a.q = q->data_ptr();
  a.k = k->data_ptr();
  a.v = v->data_ptr();
  a.o = o.data_ptr();
  a.lse = want_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
  a.q_stride_b = q->stride(0);
  a.q_stride_h = q->stride(d.h);
  a.q_stride_s = q->stride(d.s);
  a.k_stride_b = k->stride(0);
  a.k_stride_h = k->stride(d.h);
  a.k_stride_s = k->stride(d.s);
  a.v_stride_b = v->stride(0);
  a.v_stride_h = v->stride(d.h);
  a.v_stride_s = v->stride(d.s);
  a.o_stride_b = o.stride(0);
  a.o_stride_h = o.stride(d.h);
  a.o_stride_s = o.stride(d.s);
  fill_dims(a, d, causal != 0, scale, dtype, dev);
  int rc;
  if (d.Sq <= 128) {  // calls with more query rows never need a workspace
    uint64_t need = 0;
    rc = lib.fa_fwd_workspace(&a, &need);
    if (rc != HB_OK) return raise_status(rc);
    at::Tensor ws;
    if (need > 0) ws = empty_like_options(*q, {static_cast<int64_t>(need)}, at::kByte);
    rc = unlocked([&] { return lib.fa_fwd_ws(&a, need > 0 ? ws.data_ptr() : nullptr, need); });
  } else {
    rc = unlocked([&] { return lib.fa_fwd(&a); });
  }
  if (rc != HB_OK) return raise_status(rc);
  PyObject* result;
  if (args[7] != Py_None) {
    result = args[7];
    Py_INCREF(result);
  } else {
    result = THPVariable_Wrap(std::move(o));
  }
  if (!want_lse || result == nullptr) return result;
  PyObject* l = THPVariable_Wrap(std::move(lse));
  PyObject* pair = l != nullptr ? PyTuple_Pack(2, result, l) : nullptr;
  Py_DECREF(result);
  Py_XDECREF(l);
  return pair;
  END_HANDLE_TH_ERRORS
}

// fa_bwd(q, k, v, o, d_o, lse, causal, softmax_scale, layout)
PyObject* fa_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 9 || !plain_context()) return general();
  int dev;
  const at::Tensor* t[6];
  t[0] = plain_first(args[0], dev);
  if (t[0] == nullptr) return general();
  for (int i = 1; i < 6; ++i)
    if ((t[i] = plain(args[i], dev)) == nullptr) return general();
  const at::Tensor &q = *t[0], &k = *t[1], &v = *t[2], &o = *t[3], &d_o = *t[4], &lse = *t[5];
  const int layout = layout_of(args[8]), dtype = dtype16(q);
  Dims d;
  double scale;
  if (dtype < 0 || !attention_dims(q, k, layout, d) || !softmax_scale(args[7], d.D, scale)) return general();
  if (v.sizes() != k.sizes() || o.sizes() != q.sizes() || d_o.sizes() != q.sizes()) return general();
  for (int i = 2; i < 5; ++i)
    if (t[i]->scalar_type() != q.scalar_type() || t[i]->stride(3) != 1) return general();
  if (lse.dim() != 3 || lse.size(0) != d.B || lse.size(1) != d.Hq || lse.size(2) != d.Sq || !contiguous_fp32(lse, d.B * d.Hq * d.Sq)) return general();
  const int causal = PyObject_IsTrue(args[6]);
  if (causal < 0) return nullptr;
  at::Tensor delta = empty_like_options(q, {d.B, d.Hq, d.Sq}, at::kFloat);
  at::Tensor dk = empty_like_options(q, {d.B, d.Hkv, d.Skv, d.D}, q.scalar_type());
  at::Tensor dv = empty_like_options(q, {d.B, d.Hkv, d.Skv, d.D}, q.scalar_type());
  at::Tensor dq = empty_like_options(q, {d.B, d.Hq, d.Sq, d.D}, q.scalar_type());
  hb_fa_bwd_args a;
  std::memset(&a, 0, sizeof(a));
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.o = o.data_ptr();
  a.d_o = d_o.data_ptr();
  a.lse = static_cast<float*>(lse.data_ptr());
  a.delta = static_cast<float*>(delta.data_ptr());
  a.dq = dq.data_ptr();
  a.dk = dk.data_ptr();
  a.dv = dv.data_ptr();
  a.q_stride_b = q.stride(0);
  a.q_stride_h = q.stride(d.h);
  a.q_stride_s = q.stride(d.s);
  a.k_stride_b = k.stride(0);
  a.k_stride_h = k.stride(d.h);
  a.k_stride_s = k.stride(d.s);
  a.v_stride_b = v.stride(0);
  a.v_stride_h = v.stride(d.h);
  a.v_stride_s = v.stride(d.s);
  a.o_stride_b = o.stride(0);
  a.o_stride_h = o.stride(d.h);
  a.o_stride_s = o.stride(d.s);
  a.do_stride_b = d_o.stride(0);
  a.do_stride_h = d_o.stride(d.h);
  a.do_stride_s = d_o.stride(d.s);
  fill_dims(a, d, causal != 0, scale, dtype, dev);
  at::Tensor ws;
  uint64_t need = 0;
  if (d.Hq != d.Hkv) {
    const int rc = lib.fa_bwd_dkdv_workspace(&a, &need);
    if (rc != HB_OK) return raise_status(rc);
    if (need > 0) ws = empty_like_options(q, {static_cast<int64_t>(need)}, at::kByte);
  }
  const int rc = unlocked([&] { return lib.fa_bwd(&a, need > 0 ? ws.data_ptr() : nullptr, need); });
  if (rc != HB_OK) return raise_status(rc);
  if (layout == 1) {
    dq = dq.transpose(1, 2);
    dk = dk.transpose(1, 2);
    dv = dv.transpose(1, 2);
  }
  PyObject* r[3] = {THPVariable_Wrap(std::move(dq)), THPVariable_Wrap(std::move(dk)), THPVariable_Wrap(std::move(dv))};
  PyObject* all = r[0] != nullptr && r[1] != nullptr && r[2] != nullptr ? PyTuple_Pack(3, r[0], r[1], r[2]) : nullptr;
  for (PyObject* x : r) Py_XDECREF(x);
  return all;
  END_HANDLE_TH_ERRORS
}

// h2o_score(q, k, lse, causal, softmax_scale, layout)
PyObject* h2o_score(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !plain_context()) return general();
  int dev;
  const at::Tensor* q = plain_first(args[0], dev);
  if (q == nullptr) return general();
  const at::Tensor *k = plain(args[1], dev), *lse = plain(args[2], dev);
  if (k == nullptr || lse == nullptr) return general();
  const int dtype = dtype16(*q);
  Dims d;
  double scale;
  if (dtype < 0 || !attention_dims(*q, *k, layout_of(args[5]), d) || !softmax_scale(args[4], d.D, scale)) return general();
  if (lse->dim() != 3 || lse->size(0) != d.B || lse->size(1) != d.Hq || lse->size(2) != d.Sq || !contiguous_fp32(*lse, d.B * d.Hq * d.Sq)) return general();
  const int causal = PyObject_IsTrue(args[3]);
  if (causal < 0) return nullptr;
  at::Tensor score = empty_like_options(*q, {d.B, d.Hq, d.Skv}, at::kFloat);
  hb_h2o_args a;
  std::memset(&a, 0, sizeof(a));
  a.q = q->data_ptr();
  a.k = k->data_ptr();
  a.lse = static_cast<float*>(lse->data_ptr());
  a.score = static_cast<float*>(score.data_ptr());
  a.q_stride_b = q->stride(0);
  a.q_stride_h = q->stride(d.h);
  a.q_stride_s = q->stride(d.s);
  a.k_stride_b = k->stride(0);
  a.k_stride_h = k->stride(d.h);
  a.k_stride_s = k->stride(d.s);
  fill_dims(a, d, causal != 0, scale, dtype, dev);
  const int rc = unlocked([&] { return lib.h2o_score(&a); });
  if (rc != HB_OK) return raise_status(rc);
  return THPVariable_Wrap(std::move(score));
  END_HANDLE_TH_ERRORS
}

// gemm_epilogue(a, w, epilogue code, bias, row_scale, residual, rope, schedule code)
PyObject* gemm_epilogue(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t epilogue, schedule;
  if (n != 8 || !plain_context() || !integer(args[2], epilogue) || !integer(args[7], schedule)) return general();
  int dev;
  const at::Tensor* a = plain_first(args[0], dev);
  if (a == nullptr || a->dim() < 1) return general();
  const at::Tensor* w = plain(args[1], dev);
  const int dtype = dtype16(*a);
  const int64_t K = a->size(-1), M = a->numel() / K;
  if (w == nullptr || dtype < 0 || w->scalar_type() != a->scalar_type() || w->dim() != 2 || w->size(1) != K || w->stride(1) != 1) return general();
  const bool rows = a->dim() == 2 && a->stride(1) == 1;
  const int64_t N = w->size(0), n_out = epilogue == HB_EPI_SWIGLU ? N / 2 : N;
  if ((!rows && !a->is_contiguous()) || !fits_int(M) || !fits_int(N) || !fits_int(K) || n_out == 0) return general();
  hb_gemm_args g;
  std::memset(&g, 0, sizeof(g));
  if (args[3] != Py_None) {
    const at::Tensor* bias = plain(args[3], dev);
    if (bias == nullptr || bias->scalar_type() != a->scalar_type() || !bias->is_contiguous() || bias->numel() != N) return general();
    g.bias = bias->data_ptr();
  }
  if (args[4] != Py_None) {
    const at::Tensor* rs = plain(args[4], dev);
    if (rs == nullptr || !contiguous_fp32(*rs, M)) return general();
    g.row_scale = static_cast<float*>(rs->data_ptr());
  }
  if (args[5] != Py_None) {
    const at::Tensor* r = plain(args[5], dev);
    if (r == nullptr || r->scalar_type() != a->scalar_type() || !r->is_contiguous() || r->dim() < 1 || r->size(-1) != n_out || r->numel() != M * n_out)
      return general();
    g.residual = r->data_ptr();
    g.ldr = n_out;
  }
  g.dtype = dtype;
  if (epilogue == HB_EPI_ROPE) {
    if (!PyTuple_CheckExact(args[6]) || PyTuple_GET_SIZE(args[6]) != 4) return general();
    const at::Tensor *cos = plain(PyTuple_GET_ITEM(args[6], 0), dev), *sin = plain(PyTuple_GET_ITEM(args[6], 1), dev);
    int64_t head_dim, rope_cols;
    if (cos == nullptr || sin == nullptr || cos->dim() < 1 || !integer(PyTuple_GET_ITEM(args[6], 2), head_dim) ||
        !integer(PyTuple_GET_ITEM(args[6], 3), rope_cols) || !fits_int(head_dim) || !fits_int(rope_cols) || !cos->is_contiguous() || !sin->is_contiguous() ||
        std::min(cos->numel(), sin->numel()) < cos->size(0) * (head_dim / 2))
      return general();
    if (cos->scalar_type() == a->scalar_type() && sin->scalar_type() == a->scalar_type() && aligned16(*cos) && aligned16(*sin)) {
      g.dtype |= HB_GEMM_ROPE_TABLES_16;  // read as they are
    } else if (cos->scalar_type() != at::kFloat || sin->scalar_type() != at::kFloat) {
      return general();
    }
    g.rope_cos = static_cast<float*>(cos->data_ptr());
    g.rope_sin = static_cast<float*>(sin->data_ptr());
    g.rope_seq = static_cast<int32_t>(cos->size(0));
    g.head_dim = static_cast<int32_t>(head_dim);
    g.rope_cols = static_cast<int32_t>(rope_cols);
  }
  c10::SmallVector<int64_t, 6> shape(a->sizes().begin(), a->sizes().end());
  shape.back() = n_out;
  at::Tensor out = empty_like_options(*a, shape, a->scalar_type());
  g.a = a->data_ptr();
  g.w = w->data_ptr();
  g.out = out.data_ptr();
  g.M = static_cast<int32_t>(M);
  g.N = static_cast<int32_t>(N);
  g.K = static_cast<int32_t>(K);
  g.lda = rows && M > 1 ? a->stride(0) : K;  // a single row may carry any stride
  g.ldw = w->stride(0);
  g.ldo = n_out;
  g.epilogue = static_cast<int32_t>(epilogue);
  g.schedule = static_cast<int32_t>(schedule);
  g.stream = stream_of(dev);
  const int rc = unlocked([&] { return lib.gemm_epilogue(&g); });
  if (rc != HB_OK) return raise_status(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// bmm(a, b, epilogue code, schedule code)
PyObject* bmm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t epilogue, schedule;
  if (n != 4 || !plain_context() || !integer(args[2], epilogue) || !integer(args[3], schedule)) return general();
  int dev;
  const at::Tensor* a = plain_first(args[0], dev);
  if (a == nullptr) return general();
  const at::Tensor* b = plain(args[1], dev);
  const int dtype = dtype16(*a);
  if (b == nullptr || dtype < 0 || b->scalar_type() != a->scalar_type() || a->dim() != 3 || b->dim() != 3 || a->size(0) != b->size(0) ||
      a->size(2) != b->size(1))
    return general();
  const int64_t Bn = a->size(0), M = a->size(1), K = a->size(2), N = b->size(2);
  if (K % 8 || N % 8 || !fits_int(Bn) || !fits_int(M) || !fits_int(K) || !fits_int(N)) return general();
  // the library reads a batch stride of 0 as densely packed batches
  if (a->stride(2) != 1 || a->stride(1) % 8 || a->stride(0) % 8 || !aligned16(*a) || (Bn > 1 && (a->stride(0) == 0 || b->stride(0) == 0))) return general();
  if (b->stride(0) % 8 || !aligned16(*b)) return general();
  hb_gemm_args g;
  std::memset(&g, 0, sizeof(g));
  if (b->stride(1) == 1 && b->stride(2) >= K && b->stride(2) % 8 == 0 && K > 1) {
    g.w_layout = HB_W_NK;  // a transposed view of [B, N, K] storage
    g.ldw = b->stride(2);
  } else if (b->stride(2) == 1 && b->stride(1) % 8 == 0) {
    g.w_layout = HB_W_KN;
    g.ldw = b->stride(1);
  } else {
    return general();
  }
  at::Tensor out = empty_like_options(*a, {Bn, M, N}, a->scalar_type());
  g.a = a->data_ptr();
  g.w = b->data_ptr();
  g.out = out.data_ptr();
  g.M = static_cast<int32_t>(M);
  g.N = static_cast<int32_t>(N);
  g.K = static_cast<int32_t>(K);
  g.lda = a->stride(1);
  g.ldo = N;
  g.dtype = dtype;
  g.epilogue = static_cast<int32_t>(epilogue);
  g.batch = static_cast<int32_t>(Bn);
  g.a_batch_stride = a->stride(0);
  g.w_batch_stride = b->stride(0);
  g.o_batch_stride = M * N;
  g.schedule = static_cast<int32_t>(schedule);
  g.stream = stream_of(dev);
  const int rc = unlocked([&] { return lib.gemm_epilogue(&g); });
  if (rc != HB_OK) return raise_status(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// rms_rowstat(x, eps): the statistic alone
PyObject* rms_rowstat(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  double eps;
  if (n != 2 || !plain_context() || !number(args[1], eps)) return general();
  int dev;
  const at::Tensor* x = plain_first(args[0], dev);
  if (x == nullptr || x->dim() < 1 || !x->is_contiguous() || dtype16(*x) < 0) return general();
  const int64_t N = x->size(-1), M = x->numel() / N;
  if (!fits_int(N) || !fits_int(M)) return general();
  at::Tensor rstd = empty_like_options(*x, x->sizes().slice(0, x->dim() - 1), at::kFloat);
  const int rc = unlocked([&] {
    return lib.rms_rowstat(x->data_ptr(), nullptr, nullptr, static_cast<float*>(rstd.data_ptr()), static_cast<int32_t>(M), static_cast<int32_t>(N), N,
                           static_cast<float>(eps), dtype16(*x), stream_of(dev));
  });
  if (rc != HB_OK) return raise_status(rc);
  return THPVariable_Wrap(std::move(rstd));
  END_HANDLE_TH_ERRORS
}

// Rows of a (..., cols) tensor that the row kernels read in place: their stride, or -1.
int64_t row_stride(const at::Tensor& t, int64_t cols, int64_t rows) {
  if (!aligned16(t)) return -1;
  int64_t stride = cols;
  if (t.dim() == 2) {
    if (t.stride(1) != 1) return -1;
    if (rows > 1) stride = t.stride(0);  // a single row may carry any stride
  } else if (!t.is_contiguous()) {
    return -1;
  }
  return stride % 8 == 0 ? stride : -1;
}

// row_softmax(x, scale)
PyObject* row_softmax(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  double scale;
  if (n != 2 || !plain_context() || !number(args[1], scale)) return general();
  int dev;
  const at::Tensor* x = plain_first(args[0], dev);
  if (x == nullptr || x->dim() < 1 || dtype16(*x) < 0) return general();
  const int64_t cols = x->size(-1), rows = x->numel() / cols, stride = row_stride(*x, cols, rows);
  if (stride < cols || !fits_int(cols)) return general();
  at::Tensor y = empty_like_options(*x, x->sizes(), x->scalar_type());
  const int rc = unlocked([&] {
    return lib.row_softmax(x->data_ptr(), y.data_ptr(), rows, static_cast<int32_t>(cols), stride, cols, static_cast<float>(scale), dtype16(*x),
                           stream_of(dev));
  });
  if (rc != HB_OK) return raise_status(rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// Items of a list or tuple, whichever it is; false for anything else.
bool items(PyObject* o, PyObject**& first, Py_ssize_t& count) {
  if (!PyTuple_CheckExact(o) && !PyList_CheckExact(o)) return false;
  first = PySequence_Fast_ITEMS(o);
  count = PySequence_Fast_GET_SIZE(o);
  return true;
}
// The value of a name in one of _lib's tables, or -1.
int64_t named(PyObject* table, PyObject* name) {
  int64_t v;
  if (!PyUnicode_CheckExact(name)) return -1;
  PyObject* e = PyDict_GetItemWithError(table, name);
  if (e == nullptr) {
    PyErr_Clear();
    return -1;
  }
  return integer(e, v) ? v : -1;
}

// rowwise_program(program, inputs, rowvecs, rowscalars, n_outputs, mode code)
PyObject* rowwise_program(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t n_outputs, mode;
  PyObject **inst, **in, **vec, **sca;
  Py_ssize_t n_inst, n_in, n_vec, n_sca;
  if (n != 6 || !plain_context() || !items(args[0], inst, n_inst) || !items(args[1], in, n_in) || !items(args[2], vec, n_vec) ||
      !items(args[3], sca, n_sca) || !integer(args[4], n_outputs) || !integer(args[5], mode))
    return general();
  if (n_in < 1 || n_in > HB_EW_MAX_INPUTS || n_vec > HB_EW_MAX_ROWVEC || n_sca > HB_EW_MAX_ROWSCALAR || n_outputs < 1 || n_outputs > HB_EW_MAX_OUTPUTS || n_inst < 1 ||
      n_inst > HB_EW_MAX_INST)
    return general();
  hb_rowwise_args a;
  std::memset(&a, 0, sizeof(a));
  int dev;
  const at::Tensor* x0 = plain_first(in[0], dev);
  if (x0 == nullptr || x0->dim() < 1 || dtype16(*x0) < 0) return general();
  const int64_t cols = x0->size(-1), rows = x0->numel() / cols;
  if (!fits_int(cols)) return general();
  c10::SmallVector<at::Tensor, 8> keep;  // a list may lose its tensors to another thread while the lock is released
  for (Py_ssize_t i = 0; i < n_in; ++i) {
    const at::Tensor* t = plain(in[i], dev);
    if (t == nullptr || t->sizes() != x0->sizes() || t->scalar_type() != x0->scalar_type()) return general();
    a.ld_in[i] = row_stride(*t, cols, rows);
    if (a.ld_in[i] < 0) return general();
    a.inputs[i] = t->data_ptr();
    keep.push_back(*t);
  }
  for (Py_ssize_t i = 0; i < n_vec; ++i) {
    const at::Tensor* t = plain(vec[i], dev);
    if (t == nullptr || t->scalar_type() != x0->scalar_type() || !t->is_contiguous() || t->numel() != cols) return general();
    a.rowvec[i] = t->data_ptr();
    keep.push_back(*t);
  }
  for (Py_ssize_t i = 0; i < n_sca; ++i) {
    const at::Tensor* t = plain(sca[i], dev);
    if (t == nullptr || !contiguous_fp32(*t, rows)) return general();
    a.rowscalar[i] = static_cast<float*>(t->data_ptr());
    keep.push_back(*t);
  }
  for (Py_ssize_t i = 0; i < n_inst; ++i) {
    PyObject** f;
    Py_ssize_t count;
    int64_t index;
    double imm;
    // numbers proper: another object's __float__ may change the lists that are being read
    if (!items(inst[i], f, count) || count != 4 || !integer(f[2], index) || !fits_int(index) || !(PyFloat_Check(f[3]) || PyLong_CheckExact(f[3])) ||
        !number(f[3], imm))
      return general();
    const int64_t op = named(g_ew_ops, f[0]), src = f[1] == Py_None ? 0 : named(g_ew_srcs, f[1]);  // EW_SRCS["none"] is 0
    if (op < 0 || src < 0) return general();
    a.program[i].op = static_cast<int32_t>(op);
    a.program[i].src = static_cast<int32_t>(src);
    a.program[i].index = static_cast<int32_t>(index);
    a.program[i].imm = static_cast<float>(imm);
  }
  at::Tensor outs[HB_EW_MAX_OUTPUTS];
  for (int64_t i = 0; i < n_outputs; ++i) {
    outs[i] = empty_like_options(*x0, x0->sizes(), x0->scalar_type());
    a.outputs[i] = outs[i].data_ptr();
    a.ld_out[i] = cols;
  }
  a.n_inputs = static_cast<int32_t>(n_in);
  a.n_rowvec = static_cast<int32_t>(n_vec);
  a.n_rowscalar = static_cast<int32_t>(n_sca);
  a.n_outputs = static_cast<int32_t>(n_outputs);
  a.rows = rows;
  a.cols = static_cast<int32_t>(cols);
  a.dtype = dtype16(*x0);
  a.n_inst = static_cast<int32_t>(n_inst);
  a.mode = static_cast<int32_t>(mode);
  a.stream = stream_of(dev);
  const int rc = unlocked([&] { return lib.rowwise_program(&a); });
  if (rc != HB_OK) return raise_status(rc);
  if (n_outputs == 1) return THPVariable_Wrap(std::move(outs[0]));
  PyObject* all = PyTuple_New(n_outputs);
  for (int64_t i = 0; all != nullptr && i < n_outputs; ++i) {
    PyObject* t = THPVariable_Wrap(std::move(outs[i]));
    if (t == nullptr) {
      Py_DECREF(all);
      return nullptr;
    }
    PyTuple_SET_ITEM(all, i, t);
  }
  return all;
  END_HANDLE_TH_ERRORS
}

// tensors_state(tensors): storage address, version, type, device, sizes and strides of each, as bytes that are equal exactly
// where all of these are
PyObject* tensors_state(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  PyObject** t;
  Py_ssize_t count;
  if (n != 1 || !items(args[0], t, count)) return general();
  c10::SmallVector<int64_t, 64> state;
  for (Py_ssize_t i = 0; i < count; ++i) {
    if (!THPVariable_CheckExact(t[i])) return general();
    const at::Tensor& x = THPVariable_Unpack(t[i]);
    if (!x.defined() || x.layout() != at::kStrided || x.key_set().has_any(special_keys())) return general();
    state.push_back(reinterpret_cast<int64_t>(x.data_ptr()));
    state.push_back(x.is_inference() ? -1 : static_cast<int64_t>(x._version()));
    state.push_back(static_cast<int64_t>(x.scalar_type()));
    state.push_back(static_cast<int64_t>(x.device().type()) * 1024 + x.device().index());
    state.push_back(x.dim());
    state.append(x.sizes().begin(), x.sizes().end());
    state.append(x.strides().begin(), x.strides().end());
  }
  return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(state.data()), static_cast<Py_ssize_t>(state.size() * sizeof(int64_t)));
  END_HANDLE_TH_ERRORS
}

// bind(addresses by name, check, EW_OPS, EW_SRCS)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4 || !PyDict_Check(args[0]) || !PyCallable_Check(args[1]) || !PyDict_Check(args[2]) || !PyDict_Check(args[3])) {
    PyErr_SetString(PyExc_TypeError, "bind(dict, callable, dict, dict)");
    return nullptr;
  }
#define HB_BIND(name)                                                                      \
  {                                                                                        \
    PyObject* address = PyDict_GetItemString(args[0], "hb_" #name);                        \
    void* p = address != nullptr ? PyLong_AsVoidPtr(address) : nullptr;                    \
    if (p == nullptr) {                                                                    \
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, "hb_" #name);                 \
      return nullptr;                                                                      \
    }                                                                                      \
    std::memcpy(&lib.name, &p, sizeof(p));                                                 \
  }
  HB_BIND(fa_fwd)
  HB_BIND(fa_fwd_workspace)
  HB_BIND(fa_fwd_ws)
  HB_BIND(fa_bwd_dkdv_workspace)
  HB_BIND(fa_bwd)
  HB_BIND(h2o_score)
  HB_BIND(gemm_epilogue)
  HB_BIND(rms_rowstat)
  HB_BIND(row_softmax)
  HB_BIND(rowwise_program)
#undef HB_BIND
  for (int i = 1; i < 4; ++i) Py_INCREF(args[i]);
  g_check = args[1];
  g_ew_ops = args[2];
  g_ew_srcs = args[3];
  Py_RETURN_NONE;
}

#define HB_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {HB_METHOD(bind),        HB_METHOD(fa_fwd),      HB_METHOD(fa_bwd),      HB_METHOD(h2o_score),
                         HB_METHOD(gemm_epilogue), HB_METHOD(bmm),       HB_METHOD(rms_rowstat), HB_METHOD(row_softmax),
                         HB_METHOD(rowwise_program), HB_METHOD(tensors_state), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Host path of the tensor-level calls (ops.py).", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
