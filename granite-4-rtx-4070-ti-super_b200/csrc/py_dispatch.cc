// Python side of the launch interface: turns PyTorch tensors into the pointers, sizes and the
// stream that the C ABI takes, and calls it.
//
// A decode-size op is 2-6 us of device time, so what the host does per call decides how fast a step
// issued call by call can run. The same conversion written in Python (dtype, contiguity and device
// checks, set_device, current_stream, ctypes argument packing) cost 7-8 us a call: a one-row norm took
// 11.8 us of host time and takes 4.4 here, launch included, a one-row GEMM 11.5 and 3.3, a two-layer
// decode step of 26 calls 335 and 108. kernels.py keeps the names, arguments and defaults and hands
// over positionally.
//
// The entry points are bound by address (bind(), called once by kernels.py with the addresses of the
// library that capi.py loaded), so this module links against no particular build of it.
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>

#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdint>

#include "../../include/granite4_b200.h"

namespace {

struct PyErrorSet {};  // thrown after a Python exception has been set

using Types = uint64_t;  // bit per at::ScalarType
constexpr Types type_bit(at::ScalarType t) { return Types(1) << static_cast<int>(t); }
constexpr Types kAny = ~Types(0);
constexpr Types kBf16 = type_bit(at::kBFloat16) | type_bit(at::ScalarType::UInt16) | type_bit(at::kShort);
constexpr Types kF32 = type_bit(at::kFloat), kI32 = type_bit(at::kInt), kI64 = type_bit(at::kLong);
constexpr Types kU8 = type_bit(at::kByte), kI8 = type_bit(at::kChar);

// Every entry point kernels.py calls through here.
#define G4_ENTRY_POINTS(X)                                                                                      \
  X(granite4_b200_set_stream) X(granite4_prefill_embed_rows) X(granite4_kernel_embed_gather)                    \
  X(granite4_kernel_rmsnorm) X(granite4_kernel_rmsnorm_batched) X(granite4_kernel_add_rmsnorm_fp8)              \
  X(granite4_kernel_add_rmsnorm_fp8_noalloc) X(granite4_kernel_fp8_quant) X(granite4_kernel_rope)               \
  X(granite4_kernel_kv_append_int8_batched) X(granite4_prefill_rope_split_append_int8)                          \
  X(granite4_gpu_multi_rope_append) X(granite4_gpu_multi_rope) X(granite4_gpu_multi_kv_append)                  \
  X(granite4_kernel_rope_at_pos) X(granite4_kernel_rope_at_pos_batched) X(granite4_kernel_kv_append_batched)    \
  X(granite4_kernel_verify_qkv_stage) X(granite4_prefill_rope_split_append) X(granite4_kernel_rope_kv_int8_paged) \
  X(granite4_kernel_argmax_rows) X(granite4_kernel_argmax_advance) X(granite4_gpu_multi_embed)                  \
  X(granite4_kernel_multi_scatter_advance) X(granite4_kernel_attn_decode_int8_paged) X(granite4_attn_split_int8) \
  X(granite4_prefill_attention_int8) X(granite4_kernel_fp8_encode_with_amax) X(granite4_kernel_gemm_fp8)        \
  X(granite4_prefill_silu_mul) X(granite4_kernel_swiglu_fp8)

struct Api {
#define X(name) decltype(&::name) name;
  G4_ENTRY_POINTS(X)
#undef X
} api;

PyObject* bind(PyObject*, PyObject* addresses) {  // {name: address}
#define X(name)                                                                                       \
  {                                                                                                   \
    PyObject* v = PyDict_GetItemString(addresses, #name);                                             \
    if (v == nullptr) return PyErr_Format(PyExc_KeyError, "no address for %s", #name);                \
    api.name = reinterpret_cast<decltype(&::name)>(PyLong_AsVoidPtr(v));                              \
    if (PyErr_Occurred()) return nullptr;                                                             \
  }
  G4_ENTRY_POINTS(X)
#undef X
  Py_RETURN_NONE;
}

// ---- arguments ------------------------------------------------------------------------------------
const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected a tensor, got %s", Py_TYPE(o)->tp_name);
    throw PyErrorSet{};
  }
  return THPVariable_Unpack(o);
}

// A tensor whose two dimensions are an entry point's rows and columns.
const at::Tensor& matrix(PyObject* o) {
  const at::Tensor& t = tensor(o);
  if (t.dim() != 2) {
    PyErr_Format(PyExc_ValueError, "expected a matrix, got a tensor of %d dimensions", static_cast<int>(t.dim()));
    throw PyErrorSet{};
  }
  return t;
}

// Device pointer of a contiguous CUDA tensor of one of the given types (None passes through as NULL).
template <typename T = void>
T* ptr(PyObject* o, Types types = kAny) {
  if (o == Py_None) return nullptr;
  const at::Tensor& t = tensor(o);
  if (!t.is_cuda()) {
    PyErr_SetString(PyExc_ValueError, "expected a CUDA tensor: these kernels have no CPU path");
    throw PyErrorSet{};
  }
  if (!t.is_contiguous()) {
    PyErr_SetString(PyExc_ValueError, "expected a contiguous tensor");
    throw PyErrorSet{};
  }
  if (!(types & type_bit(t.scalar_type()))) {
    PyErr_Format(PyExc_TypeError, "unexpected dtype %s", c10::toString(t.scalar_type()));
    throw PyErrorSet{};
  }
  return static_cast<T*>(t.data_ptr());
}

// A float32 table: a tensor or an integer device address.
const float* table(PyObject* o) {
  if (PyLong_Check(o)) return static_cast<const float*>(PyLong_AsVoidPtr(o));
  return ptr<const float>(o, kF32);
}

long long whole(PyObject* o) {
  const long long v = PyLong_Check(o) ? PyLong_AsLongLong(o) : [&] {
    PyObject* n = PyNumber_Index(o);
    if (n == nullptr) return -1ll;
    const long long w = PyLong_AsLongLong(n);
    Py_DECREF(n);
    return w;
  }();
  if (v == -1 && PyErr_Occurred()) throw PyErrorSet{};
  return v;
}
int num(PyObject* o) { return static_cast<int>(whole(o)); }
float real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyErrorSet{};
  return static_cast<float>(v);
}

// Selects the tensor's device and torch's current stream on it for the launch.
void enter(const at::Tensor& t) {
  if (!t.is_cuda()) {
    PyErr_SetString(PyExc_ValueError, "expected a CUDA tensor: these kernels have no CPU path");
    throw PyErrorSet{};
  }
  const auto dev = t.device().index();
  if (c10::cuda::current_device() != dev) c10::cuda::set_device(dev);
  api.granite4_b200_set_stream(c10::cuda::getCurrentCUDAStream(dev).stream());
}

// Runs the launcher without the interpreter lock (a launch blocks while the stream's queue is full).
template <typename F>
PyObject* launched(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS;
  rc = f();
  Py_END_ALLOW_THREADS;
  return PyLong_FromLong(rc);
}

#define OP(name, nargs)                                                                              \
  PyObject* name##_body(PyObject* const* a);                                                         \
  PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n) {                                      \
    if (n != (nargs)) return PyErr_Format(PyExc_TypeError, #name " takes %d arguments, got %zd", (nargs), n); \
    try {                                                                                            \
      return name##_body(a);                                                                         \
    } catch (const PyErrorSet&) {                                                                    \
      return nullptr;                                                                                \
    } catch (const std::exception& e) {                                                              \
      PyErr_SetString(PyExc_RuntimeError, e.what());                                                 \
      return nullptr;                                                                                \
    }                                                                                                \
  }                                                                                                  \
  PyObject* name##_body(PyObject* const* a)

// ---- a1 -------------------------------------------------------------------------------------------
OP(prefill_embed_rows, 6) {  // tokens, start, rows, emb, mult, out
  const at::Tensor& emb = tensor(a[3]);
  enter(emb);
  const auto* tok = ptr<const int32_t>(a[0], kI32);
  const int start = num(a[1]), rows = num(a[2]), H = static_cast<int>(emb.size(-1));
  const auto* e = ptr<const uint16_t>(a[3], kBf16);
  const float mult = real(a[4]);
  auto* out = ptr<uint16_t>(a[5], kBf16);
  return launched([&] { return api.granite4_prefill_embed_rows(tok, start, rows, e, mult, out, H); });
}

OP(embed_gather, 4) {  // tokens, emb, mult, out
  const at::Tensor& emb = tensor(a[1]);
  enter(emb);
  const auto* tok = ptr<const int32_t>(a[0], kI32);
  const long long rows = tensor(a[0]).numel();
  const auto* e = ptr<const uint16_t>(a[1], kBf16);
  const float mult = real(a[2]);
  auto* out = ptr<uint16_t>(a[3], kBf16);
  const int vocab = static_cast<int>(emb.size(0)), H = static_cast<int>(emb.size(1));
  return launched([&] { return api.granite4_kernel_embed_gather(tok, rows, e, vocab, mult, out, H); });
}

// ---- a2 / a5 ----------------------------------------------------------------------------------------
OP(rmsnorm, 7) {  // x, w, eps, rows, cols, out, batched
  enter(tensor(a[0]));
  const auto* x = ptr<const uint16_t>(a[0], kBf16);
  const auto* w = ptr<const uint16_t>(a[1], kBf16);
  const float eps = real(a[2]);
  const int rows = num(a[3]), cols = num(a[4]), batched = PyObject_IsTrue(a[6]);
  auto* out = ptr<uint16_t>(a[5], kBf16);
  const auto fn = batched ? api.granite4_kernel_rmsnorm_batched : api.granite4_kernel_rmsnorm;
  return launched([&] { return fn(x, w, eps, rows, cols, out); });
}

OP(add_rmsnorm_fp8, 10) {  // y, res, w, eps, resid_mult, h_out, n_bf16, n_fp8, scale_amax, rstd
  const at::Tensor& y = matrix(a[0]);
  enter(y);
  const int rows = static_cast<int>(y.size(0)), cols = static_cast<int>(y.size(1));
  const int yf = y.scalar_type() == at::kFloat, rf = a[1] != Py_None && tensor(a[1]).scalar_type() == at::kFloat;
  const void *yp = ptr(a[0]), *rp = ptr(a[1]);
  const auto* w = ptr<const uint16_t>(a[2], kBf16);
  const float eps = real(a[3]), rm = real(a[4]);
  auto* h = ptr<uint16_t>(a[5], kBf16);
  auto* nb = ptr<uint16_t>(a[6], kBf16);
  auto* n8 = ptr<uint8_t>(a[7], kU8);
  auto* sc = ptr<float>(a[8], kF32);
  auto* rstd = ptr<float>(a[9], kF32);
  return launched(
      [&] { return api.granite4_kernel_add_rmsnorm_fp8(yp, yf, rp, rf, w, eps, rm, rows, cols, h, nb, n8, sc, rstd); });
}

OP(add_rmsnorm_fp8_noalloc, 8) {  // y, res, w, eps, resid_mult, h_out, n_fp8, scale_amax
  const at::Tensor& y = matrix(a[0]);
  enter(y);
  const int rows = static_cast<int>(y.size(0)), cols = static_cast<int>(y.size(1));
  const int yf = y.scalar_type() == at::kFloat, rf = a[1] != Py_None && tensor(a[1]).scalar_type() == at::kFloat;
  const void *yp = ptr(a[0]), *rp = ptr(a[1]);
  const auto* w = ptr<const uint16_t>(a[2], kBf16);
  const float eps = real(a[3]), rm = real(a[4]);
  auto* h = ptr<uint16_t>(a[5], kBf16);
  auto* n8 = ptr<uint8_t>(a[6], kU8);
  auto* sc = ptr<float>(a[7], kF32);
  return launched(
      [&] { return api.granite4_kernel_add_rmsnorm_fp8_noalloc(yp, yf, rp, rf, w, eps, rm, rows, cols, h, n8, sc); });
}

OP(fp8_quant, 3) {  // x, codes, scale_amax
  const at::Tensor& x = tensor(a[0]);
  enter(x);
  const auto* xp = ptr<const uint16_t>(a[0], kBf16);
  auto* c = ptr<uint8_t>(a[1], kU8);
  auto* sc = ptr<float>(a[2], kF32);
  const long long n = x.numel();
  return launched([&] { return api.granite4_kernel_fp8_quant(xp, n, c, sc); });
}

OP(fp8_encode_with_amax, 3) {  // x, codes, scale_amax
  const at::Tensor& x = tensor(a[0]);
  enter(x);
  const auto* xp = ptr<const uint16_t>(a[0], kBf16);
  auto* c = ptr<uint8_t>(a[1], kU8);
  auto* sc = ptr<float>(a[2], kF32);
  const long long n = x.numel();
  return launched([&] { return api.granite4_kernel_fp8_encode_with_amax(xp, n, c, sc); });
}

// ---- a3 -------------------------------------------------------------------------------------------
OP(rope, 6) {  // x, cos, sin, rows, head_dim, out
  enter(tensor(a[0]));
  const auto* x = ptr<const uint16_t>(a[0], kBf16);
  const float *c = table(a[1]), *s = table(a[2]);
  const int rows = num(a[3]), d = num(a[4]);
  auto* out = ptr<uint16_t>(a[5], kBf16);
  return launched([&] { return api.granite4_kernel_rope(x, c, s, rows, d, out); });
}

OP(kv_append_int8_batched, 12) {  // k, v, ck, cv, ks, vs, base_pos, rows, stride, Hk, d, pt
  enter(tensor(a[0]));
  const auto* k = ptr<const uint16_t>(a[0], kBf16);
  const auto* v = ptr<const uint16_t>(a[1], kBf16);
  auto* ck = ptr<int8_t>(a[2], kI8);
  auto* cv = ptr<int8_t>(a[3], kI8);
  auto* ks = ptr<float>(a[4], kF32);
  auto* vs = ptr<float>(a[5], kF32);
  const int base = num(a[6]), rows = num(a[7]), stride = num(a[8]), Hk = num(a[9]), d = num(a[10]);
  const auto* pt = ptr<const int>(a[11], kI32);
  return launched(
      [&] { return api.granite4_kernel_kv_append_int8_batched(k, v, ck, cv, ks, vs, base, rows, stride, Hk, d, pt); });
}

OP(prefill_rope_split_append_int8, 15) {  // qkv, cos, sin, base_pos, rows, Hq, Hk, d, stride, q_rot, ck, cv, ks, vs, pt
  enter(tensor(a[0]));
  const auto* qkv = ptr<const uint16_t>(a[0], kBf16);
  const float *c = table(a[1]), *s = table(a[2]);
  const int base = num(a[3]), rows = num(a[4]), Hq = num(a[5]), Hk = num(a[6]), d = num(a[7]), stride = num(a[8]);
  auto* q = ptr<uint16_t>(a[9], kBf16);
  auto* ck = ptr<int8_t>(a[10], kI8);
  auto* cv = ptr<int8_t>(a[11], kI8);
  auto* ks = ptr<float>(a[12], kF32);
  auto* vs = ptr<float>(a[13], kF32);
  const auto* pt = ptr<const int>(a[14], kI32);
  return launched([&] {
    return api.granite4_prefill_rope_split_append_int8(qkv, c, s, base, rows, Hq, Hk, d, stride, q, ck, cv, ks, vs, pt);
  });
}

OP(gpu_multi_rope_append, 17) {  // q, k, v, cos, sin, d_rows, rows, Hq, Hk, d, bits, ck, cv, ks, vs, stride, q_rot
  enter(tensor(a[0]));
  const auto* q = ptr<const uint16_t>(a[0], kBf16);
  const auto* k = ptr<const uint16_t>(a[1], kBf16);
  const auto* v = ptr<const uint16_t>(a[2], kBf16);
  const float *c = table(a[3]), *s = table(a[4]);
  const auto* desc = ptr<const granite4_multi_rows>(a[5]);
  const int rows = num(a[6]), Hq = num(a[7]), Hk = num(a[8]), d = num(a[9]), bits = num(a[10]), stride = num(a[15]);
  void *ck = ptr(a[11]), *cv = ptr(a[12]);
  auto* ks = ptr<float>(a[13], kF32);
  auto* vs = ptr<float>(a[14], kF32);
  auto* qr = ptr<uint16_t>(a[16], kBf16);
  return launched([&] {
    return api.granite4_gpu_multi_rope_append(q, k, v, c, s, desc, rows, Hq, Hk, d, bits, ck, cv, ks, vs, stride, qr);
  });
}

OP(gpu_multi_rope, 8) {  // x, cos, sin, d_rows, rows, heads, d, out
  enter(tensor(a[0]));
  const auto* x = ptr<const uint16_t>(a[0], kBf16);
  const float *c = table(a[1]), *s = table(a[2]);
  const auto* desc = ptr<const granite4_multi_rows>(a[3]);
  const int rows = num(a[4]), heads = num(a[5]), d = num(a[6]);
  auto* out = ptr<uint16_t>(a[7], kBf16);
  return launched([&] { return api.granite4_gpu_multi_rope(x, c, s, desc, rows, heads, d, out); });
}

OP(gpu_multi_kv_append, 12) {  // k, v, bits, ck, cv, ks, vs, d_rows, rows, stride, Hk, d
  enter(tensor(a[0]));
  const auto* k = ptr<const uint16_t>(a[0], kBf16);
  const auto* v = ptr<const uint16_t>(a[1], kBf16);
  const int bits = num(a[2]), rows = num(a[8]), stride = num(a[9]), Hk = num(a[10]), d = num(a[11]);
  void *ck = ptr(a[3]), *cv = ptr(a[4]);
  auto* ks = ptr<float>(a[5], kF32);
  auto* vs = ptr<float>(a[6], kF32);
  const auto* desc = ptr<const granite4_multi_rows>(a[7]);
  return launched(
      [&] { return api.granite4_gpu_multi_kv_append(k, v, bits, ck, cv, ks, vs, desc, rows, stride, Hk, d); });
}

OP(rope_at_pos, 6) {  // x, cos_row, sin_row, heads, d, out
  enter(tensor(a[0]));
  const auto* x = ptr<const uint16_t>(a[0], kBf16);
  const float *c = table(a[1]), *s = table(a[2]);
  const int heads = num(a[3]), d = num(a[4]);
  auto* out = ptr<uint16_t>(a[5], kBf16);
  return launched([&] { return api.granite4_kernel_rope_at_pos(x, c, s, heads, d, out); });
}

OP(rope_at_pos_batched, 7) {  // x, cos_rows, sin_rows, rows, heads, d, out
  enter(tensor(a[0]));
  const auto* x = ptr<const uint16_t>(a[0], kBf16);
  const float *c = table(a[1]), *s = table(a[2]);
  const int rows = num(a[3]), heads = num(a[4]), d = num(a[5]);
  auto* out = ptr<uint16_t>(a[6], kBf16);
  return launched([&] { return api.granite4_kernel_rope_at_pos_batched(x, c, s, rows, heads, d, out); });
}

OP(kv_append_batched, 10) {  // k, v, ck, cv, base_pos, rows, stride, Hk, d, pt
  enter(tensor(a[0]));
  const auto* k = ptr<const uint16_t>(a[0], kBf16);
  const auto* v = ptr<const uint16_t>(a[1], kBf16);
  auto* ck = ptr<uint16_t>(a[2], kBf16);
  auto* cv = ptr<uint16_t>(a[3], kBf16);
  const int base = num(a[4]), rows = num(a[5]), stride = num(a[6]), Hk = num(a[7]), d = num(a[8]);
  const auto* pt = ptr<const int>(a[9], kI32);
  return launched([&] { return api.granite4_kernel_kv_append_batched(k, v, ck, cv, base, rows, stride, Hk, d, pt); });
}

OP(verify_qkv_stage, 16) {  // q, k, v, cos, sin, base_pos, rows, Hq, Hk, d, stride, q_rot, k_rot, ck, cv, pt
  enter(tensor(a[0]));
  const auto* q = ptr<const uint16_t>(a[0], kBf16);
  const auto* k = ptr<const uint16_t>(a[1], kBf16);
  const auto* v = ptr<const uint16_t>(a[2], kBf16);
  const float *c = table(a[3]), *s = table(a[4]);
  const int base = num(a[5]), rows = num(a[6]), Hq = num(a[7]), Hk = num(a[8]), d = num(a[9]), stride = num(a[10]);
  auto* qr = ptr<uint16_t>(a[11], kBf16);
  auto* kr = ptr<uint16_t>(a[12], kBf16);
  auto* ck = ptr<uint16_t>(a[13], kBf16);
  auto* cv = ptr<uint16_t>(a[14], kBf16);
  const auto* pt = ptr<const int>(a[15], kI32);
  return launched([&] {
    return api.granite4_kernel_verify_qkv_stage(q, k, v, c, s, base, rows, Hq, Hk, d, stride, qr, kr, ck, cv, pt);
  });
}

OP(prefill_rope_split_append, 13) {  // qkv, cos, sin, base_pos, rows, Hq, Hk, d, stride, q_rot, ck, cv, pt
  enter(tensor(a[0]));
  const auto* qkv = ptr<const uint16_t>(a[0], kBf16);
  const float *c = table(a[1]), *s = table(a[2]);
  const int base = num(a[3]), rows = num(a[4]), Hq = num(a[5]), Hk = num(a[6]), d = num(a[7]), stride = num(a[8]);
  auto* q = ptr<uint16_t>(a[9], kBf16);
  auto* ck = ptr<uint16_t>(a[10], kBf16);
  auto* cv = ptr<uint16_t>(a[11], kBf16);
  const auto* pt = ptr<const int>(a[12], kI32);
  return launched([&] {
    return api.granite4_prefill_rope_split_append(qkv, c, s, base, rows, Hq, Hk, d, stride, q, ck, cv, pt);
  });
}

OP(rope_kv_int8_paged, 16) {  // qkv, cos, sin, pos_rows, kv_rows, Hq, Hk, d, stride, max_pos, k_from_bf16, q_rot, ck, cv, ks, vs
  const at::Tensor& t = tensor(a[0]);
  enter(t);
  const auto* qkv = ptr<const uint16_t>(a[0], kBf16);
  const float *c = table(a[1]), *s = table(a[2]);
  const auto* pos = ptr<const int>(a[3], kI32);
  const auto* kvr = ptr<const int>(a[4], kI32);
  const int rows = static_cast<int>(t.size(0)), Hq = num(a[5]), Hk = num(a[6]), d = num(a[7]), stride = num(a[8]);
  const int max_pos = num(a[9]), kb = num(a[10]);
  auto* q = ptr<uint16_t>(a[11], kBf16);
  auto* ck = ptr<int8_t>(a[12], kI8);
  auto* cv = ptr<int8_t>(a[13], kI8);
  auto* ks = ptr<float>(a[14], kF32);
  auto* vs = ptr<float>(a[15], kF32);
  return launched([&] {
    return api.granite4_kernel_rope_kv_int8_paged(qkv, c, s, pos, kvr, rows, Hq, Hk, d, stride, max_pos, kb, q, ck, cv,
                                                  ks, vs);
  });
}

// ---- decode-step glue -----------------------------------------------------------------------------
OP(argmax_rows, 4) {  // logits, out, d_pos, vocab_map
  const at::Tensor& t = matrix(a[0]);
  enter(t);
  const auto* x = ptr<const uint16_t>(a[0], kBf16);
  const int rows = static_cast<int>(t.size(0)), V = static_cast<int>(t.size(1));
  auto* out = ptr<int32_t>(a[1], kI32);
  auto* pos = ptr<int>(a[2], kI32);
  const auto* map = ptr<const int32_t>(a[3], kI32);
  return launched([&] { return api.granite4_kernel_argmax_rows(x, rows, V, out, pos, map); });
}

OP(argmax_advance, 3) {  // logits, d_rows, ids_out
  const at::Tensor& t = matrix(a[0]);
  enter(t);
  const auto* x = ptr<const uint16_t>(a[0], kBf16);
  const int rows = static_cast<int>(t.size(0)), V = static_cast<int>(t.size(1));
  auto* desc = ptr<granite4_multi_rows>(a[1]);
  auto* ids = ptr<int32_t>(a[2], kI32);
  return launched([&] { return api.granite4_kernel_argmax_advance(x, rows, V, desc, ids); });
}

OP(gpu_multi_embed, 5) {  // d_rows, rows, emb, mult, out
  const at::Tensor& emb = tensor(a[2]);
  enter(emb);
  const auto* desc = ptr<const granite4_multi_rows>(a[0]);
  const int rows = num(a[1]), vocab = static_cast<int>(emb.size(0)), H = static_cast<int>(emb.size(1));
  const auto* e = ptr<const uint16_t>(a[2], kBf16);
  const float mult = real(a[3]);
  auto* out = ptr<uint16_t>(a[4], kBf16);
  return launched([&] { return api.granite4_gpu_multi_embed(desc, rows, e, vocab, mult, out, H); });
}

OP(multi_scatter_advance, 2) {  // d_rows, ids
  enter(tensor(a[1]));
  auto* desc = ptr<granite4_multi_rows>(a[0]);
  const auto* ids = ptr<const int32_t>(a[1], kI32);
  return launched([&] { return api.granite4_kernel_multi_scatter_advance(desc, ids); });
}

// ---- attention --------------------------------------------------------------------------------------
OP(attn_decode_int8_paged, 17) {
  // q, ck, cv, ks, vs, row_pos, Hq, Hk, d, stride, max_len, scale, out, rows_per_group, row_pt, pt, scratch
  const at::Tensor& t = tensor(a[0]);
  enter(t);
  const auto* q = ptr<const uint16_t>(a[0], kBf16);
  const auto* ck = ptr<const int8_t>(a[1], kI8);
  const auto* cv = ptr<const int8_t>(a[2], kI8);
  const auto* ks = ptr<const float>(a[3], kF32);
  const auto* vs = ptr<const float>(a[4], kF32);
  const auto* pos = ptr<const int>(a[5], kI32);
  const int rows = static_cast<int>(t.size(0)), Hq = num(a[6]), Hk = num(a[7]), d = num(a[8]), stride = num(a[9]);
  const int max_len = num(a[10]), per = num(a[13]);
  const float scale = real(a[11]);
  auto* out = ptr<uint16_t>(a[12], kBf16);
  const auto* row_pt = reinterpret_cast<const int* const*>(ptr<const int64_t>(a[14], kI64));
  const auto* pt = ptr<const int>(a[15], kI32);
  void* scr = ptr(a[16], kU8);
  const long long bytes = a[16] == Py_None ? 0 : tensor(a[16]).numel();
  return launched([&] {
    return api.granite4_kernel_attn_decode_int8_paged(q, ck, cv, ks, vs, pos, row_pt, pt, rows, per, Hq, Hk, d, stride,
                                                      max_len, scale, scr, bytes, out);
  });
}

OP(attn_split_int8, 22) {
  // q, ck, cv, ks, vs, scale, Hq, Hk, d, stride, out, kv_base, d_pos, pt, max_len, row_pos, row_pt, row_grp, row_tbase,
  // row_tail, window, scratch
  const at::Tensor& t = tensor(a[0]);
  enter(t);
  const auto* q = ptr<const uint16_t>(a[0], kBf16);
  const auto* ck = ptr<const int8_t>(a[1], kI8);
  const auto* cv = ptr<const int8_t>(a[2], kI8);
  const auto* ks = ptr<const float>(a[3], kF32);
  const auto* vs = ptr<const float>(a[4], kF32);
  const float scale = real(a[5]);
  const int rows = static_cast<int>(t.size(0)), Hq = num(a[6]), Hk = num(a[7]), d = num(a[8]), stride = num(a[9]);
  auto* out = ptr<uint16_t>(a[10], kBf16);
  const int base = num(a[11]), max_len = num(a[14]);
  const auto* dpos = ptr<const int>(a[12], kI32);
  const auto* pt = ptr<const int>(a[13], kI32);
  const auto* row_pos = ptr<const int>(a[15], kI32);
  const auto* row_pt = reinterpret_cast<const int* const*>(ptr<const int64_t>(a[16], kI64));
  const auto* grp = ptr<const int>(a[17], kI32);
  const int ngroups = a[17] == Py_None ? 0 : static_cast<int>(tensor(a[17]).numel());
  const auto* tbase = ptr<const int>(a[18], kI32);
  const auto* tail = ptr<const int>(a[19], kI32);
  const int window = num(a[20]);
  void* scr = ptr(a[21], kU8);
  const long long bytes = a[21] == Py_None ? 0 : tensor(a[21]).numel();
  return launched([&] {
    return api.granite4_attn_split_int8(q, ck, cv, ks, vs, scale, Hq, Hk, d, base, dpos, rows, stride, scr, bytes, out,
                                        pt, max_len, row_pos, row_pt, grp, ngroups, tbase, tail, window);
  });
}

OP(prefill_attention_int8, 14) {  // q_rot, scale, Hq, Hk, d, base_pos, stride, out, ck, cv, ks, vs, pt, scratch
  const at::Tensor& t = tensor(a[0]);
  enter(t);
  const auto* q = ptr<const uint16_t>(a[0], kBf16);
  const float scale = real(a[1]);
  const int rows = static_cast<int>(t.size(0)), Hq = num(a[2]), Hk = num(a[3]), d = num(a[4]), base = num(a[5]);
  const int stride = num(a[6]);
  auto* out = ptr<uint16_t>(a[7], kBf16);
  const auto* ck = ptr<const int8_t>(a[8], kI8);
  const auto* cv = ptr<const int8_t>(a[9], kI8);
  const auto* ks = ptr<const float>(a[10], kF32);
  const auto* vs = ptr<const float>(a[11], kF32);
  const auto* pt = ptr<const int>(a[12], kI32);
  void* scr = ptr(a[13], kU8);
  const long long bytes = a[13] == Py_None ? 0 : tensor(a[13]).numel();
  return launched([&] {
    return api.granite4_prefill_attention_int8(q, scale, Hq, Hk, d, base, rows, stride, out, ck, cv, ks, vs, pt, scr,
                                               bytes);
  });
}

// ---- FP8 GEMM -----------------------------------------------------------------------------------------
// The items of any iterable, as a tuple that this object owns.
struct Items {
  PyObject* seq;
  explicit Items(PyObject* o) : seq(PySequence_Tuple(o)) {
    if (seq == nullptr) throw PyErrorSet{};
  }
  ~Items() { Py_DECREF(seq); }
  Items(const Items&) = delete;
  Items& operator=(const Items&) = delete;
  Py_ssize_t size() const { return PyTuple_GET_SIZE(seq); }
  PyObject* item(Py_ssize_t i) const { return PyTuple_GET_ITEM(seq, i); }
  PyObject* item_or_last(Py_ssize_t i) const { return item(i < size() ? i : size() - 1); }
};

OP(gemm_fp8, 10) {  // a, w, out, a_scale, w_scales, segs, residual, resid_scale, workspace, swiglu_scale_amax
  granite4_gemm_fp8_epilogue ep{};
  {
    const Items ws(a[4]), sg(a[5]);
    if (ws.size() < 1 || ws.size() > 3 || sg.size() > 2) {
      PyErr_SetString(PyExc_ValueError, "one to three weight scales, at most two segment ends");
      return nullptr;
    }
    ep.w_scale0 = real(ws.item_or_last(0));
    ep.w_scale1 = real(ws.item_or_last(1));
    ep.w_scale2 = real(ws.item_or_last(2));
    ep.seg1 = sg.size() > 0 ? num(sg.item(0)) : INT32_MAX;
    ep.seg2 = sg.size() > 1 ? num(sg.item(1)) : INT32_MAX;
  }
  const at::Tensor& A = tensor(a[0]);
  enter(A);
  const at::Tensor &W = tensor(a[1]), &out = tensor(a[2]);
  if (W.scalar_type() != at::kByte || A.scalar_type() != at::kByte || !W.is_contiguous() || A.dim() != 2 ||
      A.stride(1) != 1) {
    PyErr_SetString(PyExc_ValueError, "a_fp8 / w_fp8 must be uint8 code matrices with unit column stride");
    return nullptr;
  }
  ep.d_a_scale = ptr<const float>(a[3], kF32);
  ep.resid_scale = real(a[7]);
  ep.ldc = static_cast<int>(out.stride(0));
  int kind = GRANITE4_GEMM_OUT_BF16;
  if (a[9] != Py_None) {
    kind = GRANITE4_GEMM_OUT_SWIGLU;
    ep.d_out_bf16 = static_cast<uint16_t*>(out.data_ptr());
    ep.d_out_scale_amax = ptr<float>(a[9], kF32);
  } else if (out.scalar_type() == at::kFloat) {
    kind = GRANITE4_GEMM_OUT_F32;
    ep.d_out_f32 = static_cast<float*>(out.data_ptr());
  } else {
    ep.d_out_bf16 = static_cast<uint16_t*>(out.data_ptr());
    if (a[6] != Py_None) {
      const at::Tensor& r = tensor(a[6]);
      if (r.stride(0) != out.stride(0)) {
        PyErr_SetString(PyExc_ValueError, "the residual must have the output's row pitch");
        return nullptr;
      }
      kind = GRANITE4_GEMM_OUT_RESIDUAL;
      ep.d_residual = static_cast<const uint16_t*>(r.data_ptr());
    }
  }
  const auto* ap = static_cast<const uint8_t*>(A.data_ptr());
  const auto* wp = static_cast<const uint8_t*>(W.data_ptr());
  const int M = static_cast<int>(A.size(0)), K = static_cast<int>(A.size(1)), N = static_cast<int>(W.size(0));
  const long long lda = A.stride(0);
  void* ws = ptr(a[8], kU8);
  const long long bytes = a[8] == Py_None ? 0 : tensor(a[8]).numel();
  return launched([&] { return api.granite4_kernel_gemm_fp8(kind, ap, lda, wp, M, N, K, &ep, ws, bytes); });
}

// ---- a4 -------------------------------------------------------------------------------------------
OP(prefill_silu_mul, 4) {  // gu, I, rows, act
  enter(tensor(a[0]));
  const auto* gu = ptr<const float>(a[0], kF32);
  const int I = num(a[1]), rows = num(a[2]);
  auto* act = ptr<uint16_t>(a[3], kBf16);
  return launched([&] { return api.granite4_prefill_silu_mul(gu, I, rows, act); });
}

OP(swiglu_fp8, 6) {  // gate, up, act_bf16, act_fp8, scale_amax, ld
  const at::Tensor &g = matrix(a[0]), &u = tensor(a[1]);
  enter(g);
  const int rows = static_cast<int>(g.size(0)), I = static_cast<int>(g.size(1));
  const long long ld = a[5] == Py_None ? g.stride(0) : whole(a[5]);
  auto* ab = ptr<uint16_t>(a[2], kBf16);
  auto* a8 = ptr<uint8_t>(a[3], kU8);
  auto* sc = ptr<float>(a[4], kF32);
  const void *gp = g.data_ptr(), *up = u.data_ptr();
  const int f32 = g.scalar_type() == at::kFloat;
  return launched([&] { return api.granite4_kernel_swiglu_fp8(gp, up, f32, ld, rows, I, ab, a8, sc); });
}

// The device and stream of a tensor, for callers that go to the C ABI themselves.
OP(enter_device_of, 1) {
  enter(tensor(a[0]));
  Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", bind, METH_O, "bind({name: address}): the library's entry points"},
    FAST(prefill_embed_rows), FAST(embed_gather), FAST(rmsnorm), FAST(add_rmsnorm_fp8), FAST(add_rmsnorm_fp8_noalloc),
    FAST(fp8_quant), FAST(fp8_encode_with_amax), FAST(rope), FAST(kv_append_int8_batched),
    FAST(prefill_rope_split_append_int8), FAST(gpu_multi_rope_append), FAST(gpu_multi_rope), FAST(gpu_multi_kv_append),
    FAST(rope_at_pos), FAST(rope_at_pos_batched), FAST(kv_append_batched), FAST(verify_qkv_stage),
    FAST(prefill_rope_split_append), FAST(rope_kv_int8_paged), FAST(argmax_rows), FAST(argmax_advance),
    FAST(gpu_multi_embed), FAST(multi_scatter_advance), FAST(attn_decode_int8_paged), FAST(attn_split_int8),
    FAST(prefill_attention_int8), FAST(gemm_fp8), FAST(prefill_silu_mul), FAST(swiglu_fp8), FAST(enter_device_of),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_dispatch", "native argument conversion of kernels.py", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dispatch() { return PyModule_Create(&module); }
