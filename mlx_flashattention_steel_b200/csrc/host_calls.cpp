// The small calls of the Python front end without Python around the launch: a call of a few microseconds on the GPU was
// bound by 15 to 20 us of attribute reads, checks, allocations and ctypes conversions on the host.
//
// Every function here does what the front end's Python code does for the calls it accepts, and returns None for every
// other call, which the Python code then takes (or refuses, with its own message) from the start.  Accepted are plain
// CUDA tensors on the current device, on the current stream: no subclass, no functorch or dispatch mode, no tracing, no
// forward-mode gradient, no gradient to record.  Nothing is kept from one call to the next.
//
// Built against the installed torch's headers (build.py); links libb200fa.so beside it.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>
#include <limits>

#include "../../include/b200fa.h"

namespace {

using at::Tensor;

// The tensor inside a torch.Tensor (or Parameter) object, if it is one that the kernels may be given as it stands
const Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  static const c10::DispatchKeySet allowed({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                                            c10::DispatchKey::AutocastCUDA});
  if (!t.defined() || (t.key_set() | allowed) != allowed || !t.is_cuda() || torch::autograd::isFwGradDefined(t)) return nullptr;
  return &t;
}
bool wants_grad(const Tensor& t) { return c10::GradMode::is_enabled() && t.requires_grad(); }

// No mode is on that would see, trace or replace what the Python code does with tensors
bool plain_mode() {
  static const c10::DispatchKeySet modes({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::PreDispatch,
                                          c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode,
                                          c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchVmapMode,
                                          c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize, c10::DispatchKey::Tracer});
  return !c10::impl::tls_local_dispatch_key_set().included_.has_any(modes) && at::impl::PythonTorchFunctionTLS::stack_len() == 0;
}
bool current_device(const Tensor& t) { return t.get_device() == c10::cuda::current_device(); }
void* current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
bool same_device(const Tensor& t, const Tensor& like) { return t.get_device() == like.get_device(); }

int half_code(at::ScalarType t) { return t == at::kHalf ? B200FA_F16 : (t == at::kBFloat16 ? B200FA_BF16 : -1); }
int dtype_code(at::ScalarType t) { return t == at::kFloat ? B200FA_F32 : half_code(t); }
int pool_code(at::ScalarType t) { return t == at::kChar ? B200FA_I8 : (t == at::kFloat8_e4m3fn ? B200FA_E4M3 : half_code(t)); }

bool fits(int64_t x) { return x >= 0 && x <= std::numeric_limits<int32_t>::max(); }
// last dimension contiguous, the other strides and the base multiples of 16 bytes
bool rows_aligned(const Tensor& t) {
  const int64_t eb = static_cast<int64_t>(t.element_size()), n = t.dim();
  if (t.stride(n - 1) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return false;
  for (int64_t i = 0; i + 1 < n; ++i)
    if (t.stride(i) * eb % 16 != 0) return false;
  return true;
}
void* ptr(const Tensor& t) { return t.data_ptr(); }
void strides3(const Tensor& t, int64_t (&s)[3]) {
  for (int i = 0; i < 3; ++i) s[i] = t.stride(i);
}
Tensor like(const Tensor& t, at::IntArrayRef shape, at::ScalarType dt) { return at::empty(shape, t.options().dtype(dt)); }

// Python objects to numbers; false where Python's own conversion would be needed
bool get_int(PyObject* o, int64_t* x);
bool get_float(PyObject* o, double* x) {
  if (PyFloat_CheckExact(o)) {
    *x = PyFloat_AS_DOUBLE(o);
    return true;
  }
  int64_t i;
  if (!get_int(o, &i)) return false;
  *x = static_cast<double>(i);
  return true;
}
// None = 1 / sqrt(head_dim), which the caller has to fill in
bool get_scale(PyObject* o, double* x, bool* given) {
  *given = o != Py_None;
  return !*given || get_float(o, x);
}
bool get_int(PyObject* o, int64_t* x) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *x = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0 && *x >= std::numeric_limits<int32_t>::min() && *x <= std::numeric_limits<int32_t>::max();
}
bool get_bool(PyObject* o, bool* x) {
  if (!PyBool_Check(o)) return false;
  *x = o == Py_True;
  return true;
}

PyObject* result(const Tensor& out, const Tensor& lse) {
  PyObject* o = THPVariable_Wrap(out);
  if (o == nullptr) return nullptr;
  PyObject* l = lse.defined() ? THPVariable_Wrap(lse) : Py_NewRef(Py_None);
  if (l == nullptr) {
    Py_DECREF(o);
    return nullptr;
  }
  PyObject* t = PyTuple_Pack(2, o, l);
  Py_DECREF(o);
  Py_DECREF(l);
  return t;
}

#define NOT_HERE Py_RETURN_NONE
#define RELEASED(expr)      \
  Py_BEGIN_ALLOW_THREADS    \
  expr;                     \
  Py_END_ALLOW_THREADS

// q, k, v of a dense call, as the kernels take them without a copy
bool dense_inputs(const Tensor& q, const Tensor& k, const Tensor& v) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || !current_device(q) || !same_device(k, q) || !same_device(v, q)) return false;
  const int code = dtype_code(q.scalar_type());
  const int64_t D = q.size(3);
  if (code < 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return false;
  if (!(D == 64 || D == 128 || (D == 256 && code != B200FA_F32)) || k.size(3) != D || v.size(3) != D) return false;
  for (int i = 0; i < 4; ++i)
    if (q.size(i) <= 0 || k.size(i) <= 0 || !fits(q.size(i)) || !fits(k.size(i)) || v.size(i) != k.size(i)) return false;
  if (k.size(0) != q.size(0) || q.size(1) % k.size(1) != 0) return false;
  if (k.size(1) > 1 && (k.stride(1) == 0 || v.stride(1) == 0)) return false;      // heads broadcast: the caller's to see
  return rows_aligned(q) && rows_aligned(k) && rows_aligned(v);
}
b200fa_desc dense_desc(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, double scale, bool causal, double softcap,
                       int64_t window_left, int64_t flags) {
  b200fa_desc d;
  std::memset(&d, 0, sizeof(d));
  d.dtype = d.kv_dtype = dtype_code(q.scalar_type());
  d.B = static_cast<int32_t>(q.size(0)); d.Hq = static_cast<int32_t>(q.size(1)); d.Hkv = static_cast<int32_t>(k.size(1));
  d.N = static_cast<int32_t>(q.size(2)); d.S = static_cast<int32_t>(k.size(2)); d.D = static_cast<int32_t>(q.size(3));
  strides3(q, d.q_strides); strides3(k, d.k_strides); strides3(v, d.v_strides); strides3(o, d.o_strides);
  d.scale = static_cast<float>(scale); d.softcap = static_cast<float>(softcap);
  d.causal = causal ? 1 : 0; d.window_left = static_cast<int32_t>(window_left); d.flags = static_cast<int32_t>(flags);
  return d;
}

// fwd(q, k, v, scale, causal, softcap, window_left, want_lse, flags, record) -> (out, lse | None), or None.  record: the
// call itself (not an autograd function around it) asks, and a gradient that would have to be recorded is not for here.
PyObject* fwd_impl(PyObject* const* a, Py_ssize_t n) {
  double scale = 0., softcap;
  bool given, causal, want_lse, record;
  int64_t window_left, flags;
  if (n != 10 || !get_scale(a[3], &scale, &given) || !get_bool(a[4], &causal) || !get_float(a[5], &softcap) || !get_int(a[6], &window_left) ||
      !get_bool(a[7], &want_lse) || !get_int(a[8], &flags) || !get_bool(a[9], &record) || !plain_mode())
    NOT_HERE;
  const Tensor *q = plain(a[0]), *k = plain(a[1]), *v = plain(a[2]);
  if (q == nullptr || k == nullptr || v == nullptr || !dense_inputs(*q, *k, *v)) NOT_HERE;
  if (record && (wants_grad(*q) || wants_grad(*k) || wants_grad(*v))) NOT_HERE;
  if (!given) scale = 1.0 / std::sqrt(static_cast<double>(q->size(3)));
  void* stream = current_stream();
  c10::NoGradGuard no_grad;
  const Tensor out = like(*q, {q->size(0), q->size(1), q->size(2), q->size(3)}, q->scalar_type());
  Tensor lse, ws;
  if (want_lse) lse = like(*q, {q->size(0), q->size(1), q->size(2)}, at::kFloat);
  const b200fa_desc d = dense_desc(*q, *k, *v, out, scale, causal, softcap, window_left, flags);
  const size_t need = b200fa_fwd_workspace_bytes(&d);
  if (need > 0) ws = like(*q, {static_cast<int64_t>(need)}, at::kByte);
  int32_t st;
  RELEASED(st = b200fa_fwd(&d, ptr(*q), ptr(*k), ptr(*v), ptr(out), want_lse ? lse.data_ptr<float>() : nullptr,
                           need > 0 ? ptr(ws) : nullptr, need, stream))
  if (st != B200FA_OK) NOT_HERE;          // the Python code meets the same error and words it
  return result(out, lse);
}

// bwd(q, k, v, out, lse, dout, scale, causal, softcap, window_left, flags) -> (dq, dk, dv), or None
PyObject* bwd_impl(PyObject* const* a, Py_ssize_t n) {
  double scale, softcap;
  bool causal;
  int64_t window_left, flags;
  if (n != 11 || !get_float(a[6], &scale) || !get_bool(a[7], &causal) || !get_float(a[8], &softcap) || !get_int(a[9], &window_left) ||
      !get_int(a[10], &flags) || !plain_mode())
    NOT_HERE;
  const Tensor* t[6];
  for (int i = 0; i < 6; ++i)
    if ((t[i] = plain(a[i])) == nullptr || wants_grad(*t[i])) NOT_HERE;
  const Tensor &q = *t[0], &k = *t[1], &v = *t[2], &out = *t[3], &lse = *t[4], &dout = *t[5];
  if (!dense_inputs(q, k, v) || q.scalar_type() == at::kFloat || q.size(3) > 128) NOT_HERE;
  if (!same_device(out, q) || !same_device(lse, q) || !same_device(dout, q) || out.sizes() != q.sizes() || dout.sizes() != q.sizes() ||
      out.scalar_type() != q.scalar_type() || dout.scalar_type() != q.scalar_type() || lse.scalar_type() != at::kFloat ||
      lse.dim() != 3 || lse.size(0) != q.size(0) || lse.size(1) != q.size(1) || lse.size(2) != q.size(2) || !out.is_contiguous() ||
      !dout.is_contiguous() || !lse.is_contiguous() || !rows_aligned(out) || !rows_aligned(dout))
    NOT_HERE;
  c10::NoGradGuard no_grad;
  void* stream = current_stream();
  const Tensor dq = like(q, q.sizes(), q.scalar_type()), dk = like(q, k.sizes(), q.scalar_type()), dv = like(q, k.sizes(), q.scalar_type());
  const b200fa_desc d = dense_desc(q, k, v, out, scale, causal, softcap, window_left, flags);
  size_t need = b200fa_bwd_workspace_bytes(&d);
  if (need < 16) need = 16;
  const Tensor ws = like(q, {static_cast<int64_t>(need)}, at::kByte);
  int32_t st;
  RELEASED(st = b200fa_bwd(&d, ptr(q), ptr(k), ptr(v), ptr(out), lse.data_ptr<float>(), ptr(dout), ptr(dq), ptr(dk), ptr(dv), ptr(ws), need, stream))
  if (st != B200FA_OK) NOT_HERE;
  PyObject *x = THPVariable_Wrap(dq), *y = THPVariable_Wrap(dk), *z = THPVariable_Wrap(dv);
  PyObject* r = x != nullptr && y != nullptr && z != nullptr ? PyTuple_Pack(3, x, y, z) : nullptr;
  Py_XDECREF(x); Py_XDECREF(y); Py_XDECREF(z);
  return r;
}

// decode(q, k_pool, v_pool, table, lens, k_scale, v_scale, scale, causal, softcap, block_size, max_kv_len, want_lse, num_splits,
//        flags, max_rows) -> (out, lse | None), or None: a paged call that runs the split-KV decode kernel
PyObject* decode_impl(PyObject* const* a, Py_ssize_t n) {
  double scale = 0., softcap;
  bool given, causal, want_lse;
  int64_t block_size, max_kv_len, num_splits, flags, max_rows;
  if (n != 16) NOT_HERE;
  // First what gives back the chunks of a prefill, the other calls that come this way: too many query rows per kv head
  const Tensor* t[5];
  if ((t[0] = plain(a[0])) == nullptr || (t[1] = plain(a[1])) == nullptr || t[0]->dim() != 4 || t[1]->dim() != 4 || !get_int(a[15], &max_rows) ||
      t[0]->size(1) * t[0]->size(2) > max_rows * t[1]->size(2))
    NOT_HERE;
  if (!get_scale(a[7], &scale, &given) || !get_bool(a[8], &causal) || !get_float(a[9], &softcap) || !get_int(a[10], &block_size) ||
      !get_int(a[11], &max_kv_len) || !get_bool(a[12], &want_lse) || !get_int(a[13], &num_splits) || !get_int(a[14], &flags) ||
      !plain_mode())
    NOT_HERE;
  for (int i = 2; i < 5; ++i)
    if ((t[i] = plain(a[i])) == nullptr) NOT_HERE;
  const Tensor &q = *t[0], &kp = *t[1], &vp = *t[2], &table = *t[3], &lens = *t[4];
  if (wants_grad(q) || wants_grad(kp) || wants_grad(vp) || vp.dim() != 4 || !current_device(q)) NOT_HERE;
  const int64_t B = q.size(0), Hq = q.size(1), Nq = q.size(2), D = q.size(3), Hkv = kp.size(2);
  const int code = half_code(q.scalar_type()), kv = pool_code(kp.scalar_type());
  const bool quant = kv == B200FA_I8 || kv == B200FA_E4M3;
  if (code < 0 || kv < 0 || (!quant && kv != code) || vp.scalar_type() != kp.scalar_type() || kp.size(1) != block_size || kp.size(3) != D ||
      vp.sizes() != kp.sizes() || B <= 0 || Hq <= 0 || Nq <= 0 || Hkv <= 0 || Hq % Hkv != 0 || block_size <= 0 || block_size % 16 != 0 ||
      max_kv_len <= 0)
    NOT_HERE;
  if (table.dim() != 2 || lens.dim() != 1 || table.size(0) != B || lens.size(0) != B || table.scalar_type() != at::kInt ||
      lens.scalar_type() != at::kInt || !table.is_contiguous() || !lens.is_contiguous())
    NOT_HERE;
  for (int i = 1; i < 5; ++i)
    if (!same_device(*t[i], q)) NOT_HERE;
  if (!q.is_contiguous() || !kp.is_contiguous() || !vp.is_contiguous() || !fits(kp.size(0)) || !fits(table.size(1)) || !fits(B * Hq)) NOT_HERE;
  const Tensor *ks = nullptr, *vs = nullptr;
  bool wide_ok = Hkv <= 128;
  if (quant) {
    ks = plain(a[5]);
    vs = plain(a[6]);
    if (ks == nullptr || vs == nullptr) NOT_HERE;
    for (const Tensor* s : {ks, vs}) {
      if (s->scalar_type() != at::kHalf || s->dim() != 3 || !s->is_contiguous() || !same_device(*s, q)) NOT_HERE;
      for (int i = 0; i < 3; ++i)
        if (s->size(i) != kp.size(i)) NOT_HERE;
      wide_ok = wide_ok && reinterpret_cast<uintptr_t>(s->data_ptr()) % 16 == 0;
    }
  }
  const int64_t rows = Hq / Hkv * Nq;
  if (rows > (wide_ok ? max_rows : 8) || !(D == 128 || (D == 64 && !quant))) NOT_HERE;
  if (!given) scale = 1.0 / std::sqrt(static_cast<double>(D));
  c10::NoGradGuard no_grad;
  void* stream = current_stream();
  const Tensor out = like(q, q.sizes(), q.scalar_type());
  Tensor lse;
  if (want_lse) lse = like(q, {B, Hq, Nq}, at::kFloat);
  b200fa_desc d;
  std::memset(&d, 0, sizeof(d));
  d.dtype = code; d.kv_dtype = kv;
  d.B = static_cast<int32_t>(B); d.Hq = static_cast<int32_t>(Hq); d.Hkv = static_cast<int32_t>(Hkv); d.N = static_cast<int32_t>(Nq);
  d.D = static_cast<int32_t>(D);
  d.scale = static_cast<float>(scale); d.softcap = static_cast<float>(softcap); d.causal = causal ? 1 : 0; d.window_left = -1;
  d.num_splits = static_cast<int32_t>(num_splits);
  d.flags = static_cast<int32_t>(flags) | (rows > 8 ? B200FA_FLAG_DECODE_WIDE : 0);
  size_t need = b200fa_decode_paged_workspace_bytes(&d, static_cast<int32_t>(max_kv_len));
  if (need < 16) need = 16;
  const Tensor ws = like(q, {static_cast<int64_t>(need)}, at::kByte);
  int32_t st;
  RELEASED(st = b200fa_decode_paged(&d, ptr(q), ptr(kp), ptr(vp), quant ? ptr(*ks) : nullptr, quant ? ptr(*vs) : nullptr,
                                    table.data_ptr<int32_t>(), lens.data_ptr<int32_t>(), static_cast<int32_t>(kp.size(0)),
                                    static_cast<int32_t>(block_size), static_cast<int32_t>(table.size(1)), static_cast<int32_t>(max_kv_len),
                                    ptr(out), want_lse ? lse.data_ptr<float>() : nullptr, ptr(ws), need, stream))
  if (st != B200FA_OK) NOT_HERE;
  return result(out, lse);
}

// rope(x, cos, sin, offset, interleaved, rot | None) -> out, or None.  offset: an int, or a tuple or list of ints
PyObject* rope_impl(PyObject* const* a, Py_ssize_t n) {
  bool interleaved;
  int64_t rot = 0;
  if (n != 6 || !get_bool(a[4], &interleaved) || (a[5] != Py_None && !get_int(a[5], &rot)) || !plain_mode()) NOT_HERE;
  const Tensor *x = plain(a[0]), *cos = plain(a[1]), *sin = plain(a[2]);
  if (x == nullptr || cos == nullptr || sin == nullptr || wants_grad(*x) || wants_grad(*cos) || wants_grad(*sin)) NOT_HERE;
  if (x->dim() != 4 || !current_device(*x) || !same_device(*cos, *x) || !same_device(*sin, *x)) NOT_HERE;
  const int code = half_code(x->scalar_type());
  const int64_t B = x->size(0), H = x->size(1), N = x->size(2), D = x->size(3);
  if (a[5] == Py_None) rot = D;
  for (int i = 0; i < 4; ++i)
    if (x->size(i) <= 0 || !fits(x->size(i))) NOT_HERE;
  if (code < 0 || rot <= 0 || rot > D || rot % 2 != 0 || cos->dim() != 2 || cos->size(1) != rot / 2 || cos->sizes() != sin->sizes() ||
      cos->scalar_type() != at::kFloat || sin->scalar_type() != at::kFloat || !cos->is_contiguous() || !sin->is_contiguous() ||
      !fits(cos->size(0)) || !rows_aligned(*x))
    NOT_HERE;
  const int64_t last = cos->size(0) - N;
  int32_t offs[512];
  int64_t offset = 0;
  const bool many = !PyLong_CheckExact(a[3]);
  if (!many) {
    if (!get_int(a[3], &offset) || offset < 0 || offset > last) NOT_HERE;
  } else {
    if (!PyTuple_CheckExact(a[3]) && !PyList_CheckExact(a[3])) NOT_HERE;
    if (B > 512 || PySequence_Fast_GET_SIZE(a[3]) != B) NOT_HERE;
    PyObject** items = PySequence_Fast_ITEMS(a[3]);
    for (int64_t b = 0; b < B; ++b) {
      int64_t o;
      if (!get_int(items[b], &o) || o < 0 || o > last) NOT_HERE;
      offs[b] = static_cast<int32_t>(o);
    }
  }
  c10::NoGradGuard no_grad;
  void* stream = current_stream();
  const Tensor out = like(*x, {B, H, N, D}, x->scalar_type());
  int64_t xs[3], os[3];
  strides3(*x, xs);
  strides3(out, os);
  int32_t st;
  const int32_t b = static_cast<int32_t>(B), h = static_cast<int32_t>(H), nn = static_cast<int32_t>(N), dd = static_cast<int32_t>(D),
                r = static_cast<int32_t>(rot), mp = static_cast<int32_t>(cos->size(0));
  RELEASED(st = many ? b200fa_rope_host_offsets(code, b, h, nn, dd, r, interleaved ? 1 : 0, 0, ptr(*x), xs, ptr(out), os, cos->data_ptr<float>(),
                                                sin->data_ptr<float>(), mp, offs, stream)
                     : b200fa_rope(code, b, h, nn, dd, r, interleaved ? 1 : 0, 0, ptr(*x), xs, ptr(out), os, cos->data_ptr<float>(),
                                   sin->data_ptr<float>(), mp, nullptr, static_cast<int32_t>(offset), stream))
  if (st != B200FA_OK) NOT_HERE;
  return THPVariable_Wrap(out);
}

// append(k_new, v_new, slots, k_pool, v_pool, k_scale, v_scale) -> True, or None
PyObject* append_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 7 || !plain_mode()) NOT_HERE;
  const Tensor* t[5];
  for (int i = 0; i < 5; ++i)
    if ((t[i] = plain(a[i])) == nullptr) NOT_HERE;
  const Tensor &k = *t[0], &v = *t[1], &slots = *t[2], &kp = *t[3], &vp = *t[4];
  const int code = half_code(k.scalar_type()), kv = pool_code(kp.scalar_type());
  const bool quant = kv == B200FA_I8 || kv == B200FA_E4M3;
  if (code < 0 || kv < 0 || v.scalar_type() != k.scalar_type() || vp.scalar_type() != kp.scalar_type() || k.dim() != 3 || v.sizes() != k.sizes() ||
      kp.dim() != 4 || vp.sizes() != kp.sizes() || kp.size(2) != k.size(1) || kp.size(3) != k.size(2) || slots.scalar_type() != at::kLong ||
      slots.numel() != k.size(0) || k.size(0) <= 0 || !fits(k.size(0)) || !current_device(kp))
    NOT_HERE;
  for (int i = 0; i < 5; ++i)
    if (!same_device(*t[i], kp)) NOT_HERE;
  if (!kp.is_contiguous() || !vp.is_contiguous() || !slots.is_contiguous() || !rows_aligned(k) || !rows_aligned(v) || v.strides() != k.strides()) NOT_HERE;
  const Tensor *ks = nullptr, *vs = nullptr;
  if (quant) {
    ks = plain(a[5]);
    vs = plain(a[6]);
    if (ks == nullptr || vs == nullptr) NOT_HERE;
    for (const Tensor* s : {ks, vs}) {
      if (s->scalar_type() != at::kHalf || s->dim() != 3 || !s->is_contiguous() || !same_device(*s, kp)) NOT_HERE;
      for (int i = 0; i < 3; ++i)
        if (s->size(i) != kp.size(i)) NOT_HERE;
    }
  }
  void* stream = current_stream();
  int32_t st;
  RELEASED(st = b200fa_kv_append(code, kv, static_cast<int32_t>(k.size(0)), static_cast<int32_t>(k.size(1)), static_cast<int32_t>(k.size(2)),
                                 static_cast<int32_t>(kp.size(1)), kp.size(0), ptr(k), ptr(v), k.stride(0), k.stride(1),
                                 slots.data_ptr<int64_t>(), ptr(kp), ptr(vp), quant ? ptr(*ks) : nullptr, quant ? ptr(*vs) : nullptr, stream))
  if (st != B200FA_OK) NOT_HERE;
  Py_RETURN_TRUE;
}

// C++ exceptions (an allocation that fails) come out as Python ones
template <PyObject* (*F)(PyObject* const*, Py_ssize_t)> PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(args, n);
  END_HANDLE_TH_ERRORS
}
#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name##_impl>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(fwd), METHOD(bwd), METHOD(decode), METHOD(rope), METHOD(append), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls() {
  PyObject* m = PyModule_Create(&module);
  // the torch and Python this was built for (build.py), for the importer to compare
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", B200FA_HOST_ABI) != 0) Py_CLEAR(m);
  return m;
}
