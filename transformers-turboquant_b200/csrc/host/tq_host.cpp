// The tails of the Python entry points as native code: row views, output allocation, the current stream and the C call.
//
// A generation step of one chat is 23 us of kernels; through Python allocations (2.3 us each), stream look-ups (2.3 us)
// and 25-argument ctypes calls (2.4 us of conversions) its launches took 52 us.  The checks and dispatch of the public
// functions stay in Python; these functions see tensors that passed them.
//
// Nothing is kept between calls: outputs and scratch come from the caching allocator on the current stream (so scratch is
// safe with any number of streams and threads, and lands in the graph's pool during capture).  The GIL is released
// around the launches.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ops/empty.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAStream.h>

#include "tq_b200.h"

namespace {

PyObject* g_error = nullptr;  // turboquant_b200._lib.TurboQuantError

int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return TQ_F32;
    case at::kBFloat16: return TQ_BF16;
    case at::kHalf: return TQ_F16;
    default: return -1;
  }
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), what, " must be a tensor, got ", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}

// A [B, H, S, D] tensor whose rows the kernels can read in place: supported dtype, unit inner stride, 16-byte aligned
// rows.  Anything else is copied once.
at::Tensor rows_view(const at::Tensor& in) {
  at::Tensor t = in;
  if (dtype_code(t) < 0) {
    c10::AutoGradMode no_grad(false);
    t = t.to(at::kFloat);
  }
  const int64_t esz = t.element_size();
  bool ok = t.stride(-1) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  for (int64_t i = 0; i + 1 < t.dim(); ++i) ok = ok && (t.stride(i) * esz) % 16 == 0;
  if (ok) return t;
  c10::AutoGradMode no_grad(false);
  return t.contiguous();
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

at::Tensor make(at::IntArrayRef shape, at::ScalarType type, const at::Tensor& like) {
  return at::empty(shape, at::TensorOptions().dtype(type).device(like.device()));
}

struct Unlocked {  // the GIL is not held in its scope
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

void check(int status) {
  if (status == TQ_OK) return;
  PyObject* args = Py_BuildValue("(is)", status, tq_last_error());
  if (args != nullptr) {
    PyErr_SetObject(g_error != nullptr ? g_error : PyExc_RuntimeError, args);
    Py_DECREF(args);
  }
  throw python_error();
}

template <class T>
T* ptr(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }

void need_args(Py_ssize_t n, Py_ssize_t want) {
  TORCH_CHECK_TYPE(n == want, "expected ", want, " arguments, got ", n);
}

PyObject* set_error_type(PyObject*, PyObject* type) {
  Py_XINCREF(type);
  Py_XDECREF(g_error);
  g_error = type;
  Py_RETURN_NONE;
}

// compress(keys | None, values | None, constants, bits, mode)
//   -> (key indices, signs, residual norms, norms, value indices, norms), None for a side that is not there
PyObject* compress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 5);
  at::Tensor k, v;
  if (a[0] != Py_None) k = rows_view(tensor(a[0], "keys"));
  if (a[1] != Py_None) v = rows_view(tensor(a[1], "values"));
  if (k.defined() && v.defined() && v.scalar_type() != k.scalar_type()) {
    c10::AutoGradMode no_grad(false);
    v = v.to(k.scalar_type());
  }
  const at::Tensor& x = k.defined() ? k : v;
  const at::Tensor& consts = tensor(a[2], "constants");
  const int64_t bits = integer(a[3]), mode = integer(a[4]);
  const int64_t B = x.size(0), H = x.size(1), S = x.size(2), D = x.size(3), rows = B * H * S;
  at::Tensor ki, ks, rn, vn, vi, vv;
  if (k.defined()) {
    ki = make({rows, D * (bits - 1) / 8}, at::kByte, x);
    ks = make({rows, D / 8}, at::kByte, x);
    rn = make({B, H, S}, at::kHalf, x);
    vn = make({B, H, S}, at::kHalf, x);
  }
  if (v.defined()) {
    vi = make({rows, D * bits / 8}, at::kByte, x);
    vv = make({rows}, at::kHalf, x);
  }
  int status;
  {
    void* const stream = stream_of(x);
    const bool hk = k.defined(), hv = v.defined();
    Unlocked unlocked;
    status = tq_compress_kv(
        hk ? k.data_ptr() : nullptr, hv ? v.data_ptr() : nullptr, dtype_code(x), B, H, S, (int)D, hk ? k.stride(0) : 0,
        hk ? k.stride(1) : 0, hk ? k.stride(2) : D, hv ? v.stride(0) : 0, hv ? v.stride(1) : 0, hv ? v.stride(2) : D,
        consts.data_ptr(), (int)bits, hk ? ptr<uint8_t>(ki) : nullptr, hk ? ptr<uint8_t>(ks) : nullptr,
        hk ? ptr<uint16_t>(vn) : nullptr, hk ? ptr<uint16_t>(rn) : nullptr, hv ? ptr<uint8_t>(vi) : nullptr,
        hv ? ptr<uint16_t>(vv) : nullptr, S, 0, (int)mode, stream);
  }
  check(status);
  PyObject* out = PyTuple_New(6);
  if (out == nullptr) throw python_error();
  at::Tensor* parts[6] = {&ki, &ks, &rn, &vn, &vi, &vv};
  for (int i = 0; i < 6; ++i) PyTuple_SET_ITEM(out, i, THPVariable_Wrap(std::move(*parts[i])));  // undefined -> None
  return out;
  END_HANDLE_TH_ERRORS
}

// append(keys, values, constants, bits, mode, key indices, signs, norms, residual norms, value indices, norms, capacity,
//        offset)
PyObject* append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 13);
  at::Tensor k = rows_view(tensor(a[0], "keys")), v = rows_view(tensor(a[1], "values"));
  if (v.scalar_type() != k.scalar_type()) {
    c10::AutoGradMode no_grad(false);
    v = v.to(k.scalar_type());
  }
  const at::Tensor& consts = tensor(a[2], "constants");
  const int64_t bits = integer(a[3]), mode = integer(a[4]), capacity = integer(a[11]), offset = integer(a[12]);
  void* buf[6];
  for (int i = 0; i < 6; ++i) buf[i] = tensor(a[5 + i], "cache buffer").data_ptr();
  int status;
  {
    void* const stream = stream_of(k);
    Unlocked unlocked;
    status = tq_compress_kv(k.data_ptr(), v.data_ptr(), dtype_code(k), k.size(0), k.size(1), k.size(2), (int)k.size(3),
                            k.stride(0), k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2), consts.data_ptr(),
                            (int)bits, static_cast<uint8_t*>(buf[0]), static_cast<uint8_t*>(buf[1]),
                            static_cast<uint16_t*>(buf[2]), static_cast<uint16_t*>(buf[3]), static_cast<uint8_t*>(buf[4]),
                            static_cast<uint16_t*>(buf[5]), capacity, offset, (int)mode, stream);
  }
  check(status);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// attend(q, KV heads, keys in use, capacity, (6 packed arrays), constants, bits, scale, causal, mode, mask | None, mask kind)
//   -> [B, Hq, Sq, D] in q's dtype
PyObject* attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 12);
  const at::Tensor q = rows_view(tensor(a[0], "q"));
  const int64_t Hkv = integer(a[1]), Sk = integer(a[2]), capacity = integer(a[3]);
  TORCH_CHECK_TYPE(PyTuple_Check(a[4]) && PyTuple_GET_SIZE(a[4]) == 6, "expected six packed arrays");
  const void* p[6];
  for (int i = 0; i < 6; ++i) p[i] = tensor(PyTuple_GET_ITEM(a[4], i), "packed array").data_ptr();
  const at::Tensor& consts = tensor(a[5], "constants");
  const int bits = (int)integer(a[6]), causal = (int)integer(a[8]), mode = (int)integer(a[9]);
  const float scale = (float)real(a[7]);
  const int64_t B = q.size(0), Hq = q.size(1), Sq = q.size(2), D = q.size(3);
  // [B, Hq, Sq, D] as a view of a [B, Sq, Hq, D] buffer: the adapters' `out.transpose(1, 2).reshape(B, Sq, Hq * D)` in
  // front of the output projection is then a view, not a copy (the kernels write through the strides)
  at::Tensor out = make({B, Sq, Hq, D}, q.scalar_type(), q).transpose(1, 2);
  at::Tensor mask;
  size_t need;
  if (a[10] != Py_None) {
    mask = tensor(a[10], "mask");
    need = tq_attention_masked_workspace_bytes(B, Hq, Sq, Hkv, Sk, capacity, (int)D, mode, mask.size(0));
  } else {
    need = tq_attention_prepared_workspace_bytes(B, Hq, Sq, Hkv, Sk, capacity, (int)D, mode);
  }
  at::Tensor ws;
  if (need > 0) ws = make({(int64_t)need}, at::kByte, q);
  void* const wp = need > 0 ? ws.data_ptr() : nullptr;
  const int kind = mask.defined() ? (int)integer(a[11]) : 0;
  int status;
  {
    void* const stream = stream_of(q);
    const uint8_t *ki = static_cast<const uint8_t*>(p[0]), *ks = static_cast<const uint8_t*>(p[1]);
    const uint16_t *kn = static_cast<const uint16_t*>(p[2]), *kr = static_cast<const uint16_t*>(p[3]);
    const uint8_t* vi = static_cast<const uint8_t*>(p[4]);
    const uint16_t* vn = static_cast<const uint16_t*>(p[5]);
    Unlocked unlocked;
    status = mask.defined()
                 ? tq_attention_fwd_masked(q.data_ptr(), dtype_code(q), B, Hq, Sq, (int)D, q.stride(0), q.stride(1),
                                           q.stride(2), Hkv, Sk, capacity, ki, ks, kn, kr, vi, vn, consts.data_ptr(), bits,
                                           scale, causal, mask.data_ptr(), kind, mask.size(0), mask.stride(0),
                                           mask.stride(1), out.data_ptr(), out.stride(0), out.stride(1), out.stride(2), wp,
                                           need, mode, stream)
                 : tq_attention_fwd_prepared(q.data_ptr(), dtype_code(q), B, Hq, Sq, (int)D, q.stride(0), q.stride(1),
                                             q.stride(2), Hkv, Sk, capacity, ki, ks, kn, kr, vi, vn, consts.data_ptr(), bits,
                                             scale, causal, nullptr, 0, 0, out.data_ptr(), out.stride(0), out.stride(1),
                                             out.stride(2), wp, need, mode, stream);
  }
  check(status);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// scores(q, KV heads, keys, key indices, signs, norms, residual norms, Pi, S_eff, centroids, bits) -> fp32 [B, Hq, Sq, Sk]
PyObject* scores(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 11);
  const at::Tensor q = rows_view(tensor(a[0], "queries"));
  const int64_t Hkv = integer(a[1]), Sk = integer(a[2]);
  const void* p[7];
  for (int i = 0; i < 7; ++i) p[i] = tensor(a[3 + i], "compressed keys").data_ptr();
  const int bits = (int)integer(a[10]);
  const int64_t B = q.size(0), Hq = q.size(1), Sq = q.size(2), D = q.size(3);
  at::Tensor out = make({B, Hq, Sq, Sk}, at::kFloat, q);
  const size_t need = tq_attention_workspace_bytes(B, Hq, Sq, (int)D, TQ_MODE_FP32);
  at::Tensor ws = make({(int64_t)(need > 0 ? need : 256)}, at::kByte, q);
  int status;
  {
    void* const stream = stream_of(q);
    Unlocked unlocked;
    status = tq_attention_scores(q.data_ptr(), dtype_code(q), B, Hq, Sq, (int)D, q.stride(0), q.stride(1), q.stride(2), Hkv,
                                 Sk, static_cast<const uint8_t*>(p[0]), static_cast<const uint8_t*>(p[1]),
                                 static_cast<const uint16_t*>(p[2]), static_cast<const uint16_t*>(p[3]),
                                 static_cast<const float*>(p[4]), static_cast<const float*>(p[5]),
                                 static_cast<const float*>(p[6]), bits, ptr<float>(out), ws.data_ptr(), ws.numel(),
                                 TQ_MODE_FP32, stream);
  }
  check(status);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// decompress(value indices, norms, Pi, centroids, bits, (B, H, S, D)) -> fp32 [B, H, S, D]
PyObject* decompress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 9);
  const at::Tensor& idx = tensor(a[0], "compressed values");
  const at::Tensor &vn = tensor(a[1], "norms"), &pi = tensor(a[2], "Pi"), &cen = tensor(a[3], "centroids");
  const int bits = (int)integer(a[4]);
  const int64_t B = integer(a[5]), H = integer(a[6]), S = integer(a[7]), D = integer(a[8]);
  at::Tensor out = make({B, H, S, D}, at::kFloat, idx);
  int status;
  {
    void* const stream = stream_of(idx);
    Unlocked unlocked;
    status = tq_decompress_values(ptr<const uint8_t>(idx), ptr<const uint16_t>(vn), B * H * S, (int)D, ptr<const float>(pi),
                                  ptr<const float>(cen), bits, ptr<float>(out), stream);
  }
  check(status);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// rope(q, k, cos, sin) -> (q, k) rotated, contiguous; None when the kernel does not cover these tensors: it wants CUDA
// tensors of one dtype it knows, rotary width = head_dim (a multiple of 32), cos / sin [B or 1, S, d], contiguous rows
bool rope_covers(const at::Tensor& q, const at::Tensor& k, const at::Tensor& c, const at::Tensor& s) {
  if (!q.is_cuda() || dtype_code(q) < 0 || q.dim() != 4 || k.dim() != 4 || c.dim() != 3) return false;
  const int64_t d = q.size(3);
  return k.scalar_type() == q.scalar_type() && c.scalar_type() == q.scalar_type() && s.scalar_type() == q.scalar_type() &&
         c.sizes() == s.sizes() && c.size(2) == d && d % 32 == 0 && (c.size(0) == 1 || c.size(0) == q.size(0)) &&
         c.size(1) == q.size(2) && k.size(3) == d && k.size(2) == q.size(2) && q.stride(3) == 1 && k.stride(3) == 1;
}
PyObject* py_rope_covers(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 4);
  if (rope_covers(tensor(a[0], "q"), tensor(a[1], "k"), tensor(a[2], "cos"), tensor(a[3], "sin"))) Py_RETURN_TRUE;
  Py_RETURN_FALSE;
  END_HANDLE_TH_ERRORS
}
PyObject* rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 4);
  const at::Tensor &q = tensor(a[0], "q"), &k = tensor(a[1], "k");
  at::Tensor c = tensor(a[2], "cos"), s = tensor(a[3], "sin");
  if (!rope_covers(q, k, c, s)) Py_RETURN_NONE;
  if (c.stride(-1) != 1 || s.strides() != c.strides()) {
    c10::AutoGradMode no_grad(false);
    c = c.contiguous();
    s = s.contiguous();
  }
  const int64_t B = q.size(0), Hq = q.size(1), S = q.size(2), d = q.size(3), Hkv = k.size(1);
  at::Tensor qo = make({B, Hq, S, d}, q.scalar_type(), q), ko = make({B, Hkv, S, d}, k.scalar_type(), k);
  int status;
  {
    void* const stream = stream_of(q);
    Unlocked unlocked;
    status = tq_rope(q.data_ptr(), k.data_ptr(), dtype_code(q), B, Hq, Hkv, S, (int)d, q.stride(0), q.stride(1), q.stride(2),
                     k.stride(0), k.stride(1), k.stride(2), c.data_ptr(), s.data_ptr(), c.size(0) == 1 ? 0 : c.stride(0),
                     c.stride(1), qo.data_ptr(), ko.data_ptr(), stream);
  }
  check(status);
  PyObject* pair = PyTuple_New(2);
  if (pair == nullptr) throw python_error();
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(qo)));
  PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(ko)));
  return pair;
  END_HANDLE_TH_ERRORS
}

#define TQ_FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"set_error_type", set_error_type, METH_O, nullptr},
                         TQ_FAST("compress", compress),
                         TQ_FAST("append", append),
                         TQ_FAST("attend", attend),
                         TQ_FAST("scores", scores),
                         TQ_FAST("decompress", decompress),
                         TQ_FAST("rope_covers", py_rope_covers),
                         TQ_FAST("rope", rope),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tq_host", "Native tails of the Python entry points.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tq_host() { return PyModule_Create(&module); }
