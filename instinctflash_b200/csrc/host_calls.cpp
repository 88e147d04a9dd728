// Call path from Python tensors to the C ABI of libiflb200.so.
//
// The operators of this package are called once per kernel; checking a dozen tensor attributes and
// marshalling twenty arguments from Python cost 14 to 20 us per operator, several times the kernel
// itself (attention merge of 50 tokens: 15.6 us per call for a 4.5 us kernel; a projection module,
// three kernels and four allocations: 55 us for 10 us).  Here the same attributes are read from the
// tensor objects directly and the entry point is called through its address, about 1 us beside the
// launch itself.
//
// Every function takes its operator's arguments in order, and answers True when it has launched and
// False when the arguments are not the plain accepted case: a wrong type, shape, stride or dtype, a
// tensor subclass, another device than the current one.  It never launches for arguments the Python
// operator would refuse; that operator then runs its own checks, raises its own message, or switches
// the device and launches.  A status other than 0 from the library raises RuntimeError.
//
// The library is not linked: bind() receives the addresses from the one loader of this package.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <algorithm>
#include <cmath>

#include "../../include/iflb200.h"

namespace {

#define IFLB200_CALLS(X)                                                                                        \
  X(status_string) X(row_quant) X(quant_from_amax) X(dequant_rows) X(gated_act_quant) X(residual_norm_quant)    \
  X(residual_norm_quant_partials) X(qkv_split) X(wan_qkv) X(attn_combine_quant) X(gemm_fp8_raw)                 \
  X(gemm_fp8_partials) X(fp8_linear) X(fp8_linear_residual) X(fp8_linear_gated) X(pack_workspace_bytes)         \
  X(dynamic_pack_bf16_e4m3) X(pack_bf16_e4m3)

struct Api {
#define IFLB200_FIELD(name) decltype(&iflb200_##name) name = nullptr;
  IFLB200_CALLS(IFLB200_FIELD)
#undef IFLB200_FIELD
  bool bound = false;
} api;

using at::ScalarType;
using Args = PyObject* const*;

// ------------------------------------------------------------------------------------------------
// Operands.  `ok` turns false at the first argument that is not the plain case; `dev` is the device
// of the first tensor, which every other one has to share and which has to be the current one.
// ------------------------------------------------------------------------------------------------
struct Mat {
  void* p = nullptr;
  int64_t rows = 0, cols = 0, ld = 0;
  ScalarType type = ScalarType::Undefined;
};

constexpr unsigned bit(ScalarType t) { return 1u << (unsigned)t; }
static_assert((unsigned)ScalarType::Float8_e4m3fn < 32, "type sets are 32-bit masks");
constexpr unsigned kFloats = bit(ScalarType::Float) | bit(ScalarType::BFloat16) | bit(ScalarType::Half);
constexpr unsigned kCodes = bit(ScalarType::Float8_e4m3fn);

int code_of(ScalarType t) { return t == ScalarType::Float ? IFLB200_F32 : (t == ScalarType::BFloat16 ? IFLB200_BF16 : IFLB200_F16); }

struct Call {
  bool ok = api.bound;
  int dev = -1;

  // The tensor behind `o` when it is an ordinary CUDA tensor on the call's device, else null.
  const at::Tensor* tensor(PyObject* o) {
    if (!ok) return nullptr;
    ok = false;
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != c10::kStrided || !t.has_storage() ||
        t.key_set().has(c10::DispatchKey::Python))
      return nullptr;
    const int index = t.get_device();
    if (dev < 0) dev = index;
    if (index != dev || (unsigned)t.scalar_type() >= 32) return nullptr;
    ok = true;
    return &t;
  }

  // [rows, width], contiguous rows
  Mat mat(PyObject* o, unsigned types, int64_t rows = -1, int64_t cols = -1) {
    Mat m;
    const at::Tensor* t = tensor(o);
    if (!t) return m;
    m.type = t->scalar_type();
    ok = t->dim() == 2 && (types & bit(m.type)) && (t->size(1) <= 1 || t->stride(1) == 1) &&
         (rows < 0 || t->size(0) == rows) && (cols < 0 || t->size(1) == cols) && t->size(0) <= INT32_MAX &&
         t->size(1) <= INT32_MAX;
    if (!ok) return m;
    m.rows = t->size(0);
    m.cols = t->size(1);
    m.ld = m.rows > 1 ? t->stride(0) : std::max(t->stride(0), m.cols);
    m.p = t->data_ptr();
    return m;
  }

  // optional contiguous vector of at least n elements (n < 0: any number); null pointer for None
  void* vec(PyObject* o, int64_t n, ScalarType type = ScalarType::Float, int64_t* numel = nullptr) {
    if (o == Py_None) return nullptr;
    const at::Tensor* t = tensor(o);
    if (!t) return nullptr;
    ok = t->scalar_type() == type && t->is_contiguous() && t->numel() >= n;
    if (numel) *numel = t->numel();
    return ok ? t->data_ptr() : nullptr;
  }
  float* f32(PyObject* o, int64_t n) { return static_cast<float*>(vec(o, n)); }
  // the same, but it has to be there
  float* need(PyObject* o, int64_t n) {
    if (o == Py_None) ok = false;
    return f32(o, n);
  }

  int integer(PyObject* o) {
    if (!ok) return 0;
    const long v = PyLong_Check(o) ? PyLong_AsLong(o) : -1;
    if (!PyLong_Check(o) || v < INT32_MIN || v > INT32_MAX || PyErr_Occurred()) {
      PyErr_Clear();
      ok = false;
    }
    return (int)v;
  }
  double real(PyObject* o) {
    if (!ok) return 0.0;
    const double v = PyFloat_Check(o) ? PyFloat_AS_DOUBLE(o) : (PyLong_Check(o) ? PyLong_AsDouble(o) : NAN);
    if (PyErr_Occurred()) PyErr_Clear();
    ok = v == v;
    return v;
  }
  int flag(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) {
      PyErr_Clear();
      ok = false;
    }
    return v > 0;
  }

  // ready to launch: the operands' device is the current one
  bool ready() { return ok && dev >= 0 && c10::cuda::current_device() == dev; }
  void* stream() { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }
};

PyObject* failed(int status, const char* what) {
  PyErr_Format(PyExc_RuntimeError, "%s failed with status %d: %s", what, status, api.status_string(status));
  return nullptr;
}

// The interpreter lock is given up around launches (they can wait for room in the GPU's queue) and allocations.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

template <typename F>
int unlocked(F&& call) {
  NoGil released;
  return call();
}

template <typename F>
PyObject* finish(const char* what, F&& call) {
  const int status = unlocked(call);
  if (status != 0) return failed(status, what);
  Py_RETURN_TRUE;
}

#define ARITY(n)                                                                              \
  if (nargs != (n)) {                                                                         \
    PyErr_Format(PyExc_TypeError, "%s takes %d arguments, got %zd", __func__, (n), nargs);    \
    return nullptr;                                                                           \
  }

bool gemm_shapes(const Mat& a, const Mat& w) { return a.cols == w.cols && a.cols % 16 == 0 && w.rows % 16 == 0; }

// ------------------------------------------------------------------------------------------------
// GEMM and its fused forms
// ------------------------------------------------------------------------------------------------
PyObject* gemm(PyObject*, Args v, Py_ssize_t nargs) {  // a, w, out
  ARITY(3);
  Call c;
  const Mat a = c.mat(v[0], kCodes), w = c.mat(v[1], kCodes), o = c.mat(v[2], bit(ScalarType::BFloat16), a.rows, w.rows);
  if (!c.ready() || !gemm_shapes(a, w)) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("gemm_fp8_raw", [&] {
    return api.gemm_fp8_raw(a.p, a.ld, w.p, w.ld, (int)a.rows, (int)w.rows, (int)a.cols, o.p, o.ld, s);
  });
}

PyObject* fp8_linear(PyObject*, Args v, Py_ssize_t nargs) {  // a, a_scale, w, w_scale, bias, out, exact
  ARITY(7);
  Call c;
  const Mat a = c.mat(v[0], kCodes), w = c.mat(v[2], kCodes), o = c.mat(v[5], kFloats, a.rows, w.rows);
  int64_t nr = 0, nc = 0, nb = 0;
  const float* rs = static_cast<float*>(c.vec(v[1], 0, ScalarType::Float, &nr));
  const float* cs = static_cast<float*>(c.vec(v[3], 0, ScalarType::Float, &nc));
  const void* b = nullptr;
  int bias_type = IFLB200_F32;
  if (v[4] != Py_None) {
    const at::Tensor* t = c.tensor(v[4]);
    if (!t) Py_RETURN_FALSE;
    const ScalarType bt = t->scalar_type();
    if (bt != ScalarType::Float && bt != ScalarType::BFloat16) Py_RETURN_FALSE;
    bias_type = code_of(bt);
    b = c.vec(v[4], w.rows, bt, &nb);
  }
  const int exact = c.flag(v[6]);
  if (!c.ready() || !gemm_shapes(a, w) || (b && nb != w.rows) || (rs && nr != 1 && nr != a.rows) ||
      (cs && nc != 1 && nc != w.rows))
    Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("fp8_linear", [&] {
    return api.fp8_linear(a.p, a.ld, w.p, w.ld, (int)a.rows, (int)w.rows, (int)a.cols, rs, rs && nr == 1 && a.rows != 1 ? 0 : 1,
                          cs, cs && nc == 1 && w.rows != 1 ? 0 : 1, b, bias_type,
                          exact ? IFLB200_ROUND_EXACT : IFLB200_ROUND_ENGINE, o.p, code_of(o.type), o.ld, s);
  });
}

PyObject* fp8_linear_residual(PyObject*, Args v, Py_ssize_t nargs) {  // a, a_scale, w, w_scale, bias, gate, gate_index, res
  ARITY(8);
  Call c;
  const Mat a = c.mat(v[0], kCodes), w = c.mat(v[2], kCodes);
  const Mat r = c.mat(v[7], bit(ScalarType::Float) | bit(ScalarType::BFloat16), a.rows, w.rows);
  const float* rs = c.f32(v[1], a.rows);
  const float* cs = c.f32(v[3], w.rows);
  const float* b = c.f32(v[4], w.rows);
  const float* g = c.f32(v[5], w.rows);
  const void* gi = c.vec(v[6], a.rows, ScalarType::Int);
  if (!c.ready() || !gemm_shapes(a, w)) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("fp8_linear_residual", [&] {
    return api.fp8_linear_residual(a.p, a.ld, w.p, w.ld, (int)a.rows, (int)w.rows, (int)a.cols, rs, cs, b, g,
                                   static_cast<const int32_t*>(gi), r.p, code_of(r.type), r.ld, s);
  });
}

PyObject* fp8_linear_gated(PyObject*, Args v, Py_ssize_t nargs) {  // a, a_scale, w, w_scale, h, amax, act
  ARITY(7);
  Call c;
  const Mat a = c.mat(v[0], kCodes), w = c.mat(v[2], kCodes);
  if (w.rows % 2) Py_RETURN_FALSE;
  const int64_t F = w.rows / 2;
  const Mat h = c.mat(v[4], bit(ScalarType::Float), a.rows, F);
  const float* rs = c.f32(v[1], a.rows);
  const float* cs = c.f32(v[3], w.rows);
  float* amax = c.need(v[5], a.rows);
  const int act = c.integer(v[6]);
  if (!c.ready() || a.cols != w.cols || a.cols % 16 || F % 16 || (act != 0 && act != 1)) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("fp8_linear_gated", [&] {
    return api.fp8_linear_gated(a.p, a.ld, w.p, w.ld, (int)a.rows, (int)F, (int)a.cols, rs, cs, act, static_cast<float*>(h.p),
                                h.ld, reinterpret_cast<uint32_t*>(amax), s);
  });
}

PyObject* gemm_partials(PyObject*, Args v, Py_ssize_t nargs) {  // a, w, out [S, M, N]
  ARITY(3);
  Call c;
  const Mat a = c.mat(v[0], kCodes), w = c.mat(v[1], kCodes);
  const at::Tensor* o = c.tensor(v[2]);
  if (!o || !c.ready() || !gemm_shapes(a, w) || a.cols % 128 || o->scalar_type() != ScalarType::Float ||
      o->dim() != 3 || o->size(1) != a.rows || o->size(2) != w.rows || !o->is_contiguous() || o->size(0) > 1024)
    Py_RETURN_FALSE;
  float* out = static_cast<float*>(o->data_ptr());
  const int splits = (int)o->size(0);
  void* s = c.stream();
  return finish("gemm_fp8_partials", [&] {
    return api.gemm_fp8_partials(a.p, a.ld, w.p, w.ld, (int)a.rows, (int)w.rows, (int)a.cols, splits, out, w.rows, s);
  });
}

// ------------------------------------------------------------------------------------------------
// Row operators
// ------------------------------------------------------------------------------------------------
PyObject* row_quant(PyObject*, Args v, Py_ssize_t nargs) {  // x, q, q_scale, row, col, bias, gelu
  ARITY(7);
  Call c;
  const Mat x = c.mat(v[0], kFloats), q = c.mat(v[1], kCodes, x.rows, x.cols);
  float* qs = c.need(v[2], x.rows);
  const float* row = c.f32(v[3], x.rows);
  const float* col = c.f32(v[4], x.cols);
  const float* bias = c.f32(v[5], x.cols);
  const int gelu = c.flag(v[6]);
  if (!c.ready()) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("row_quant", [&] {
    return api.row_quant(x.p, code_of(x.type), x.ld, (int)x.rows, (int)x.cols, row, col, bias, gelu, q.p, q.ld, qs, s);
  });
}

PyObject* quant_from_amax(PyObject*, Args v, Py_ssize_t nargs) {  // h, amax, q, q_scale, zero
  ARITY(5);
  Call c;
  const Mat h = c.mat(v[0], bit(ScalarType::Float)), q = c.mat(v[2], kCodes, h.rows, h.cols);
  const float* amax = c.need(v[1], h.rows);
  float* qs = c.need(v[3], h.rows);
  float* zero = c.f32(v[4], h.rows);
  if (!c.ready() || zero == amax) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("quant_from_amax", [&] {
    return api.quant_from_amax(static_cast<const float*>(h.p), h.ld, (int)h.rows, (int)h.cols, amax, zero, q.p, q.ld, qs, s);
  });
}

PyObject* dequant_rows(PyObject*, Args v, Py_ssize_t nargs) {  // x, y, row, col, bias
  ARITY(5);
  Call c;
  const Mat x = c.mat(v[0], kFloats), y = c.mat(v[1], kFloats, x.rows, x.cols);
  const float* row = c.f32(v[2], x.rows);
  const float* col = c.f32(v[3], x.cols);
  const float* bias = c.f32(v[4], x.cols);
  if (!c.ready()) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("dequant_rows", [&] {
    return api.dequant_rows(x.p, code_of(x.type), x.ld, (int)x.rows, (int)x.cols, row, col, bias, y.p, code_of(y.type), y.ld, s);
  });
}

PyObject* gated_act_quant(PyObject*, Args v, Py_ssize_t nargs) {  // gu, q, q_scale, row, col, act
  ARITY(6);
  Call c;
  const Mat gu = c.mat(v[0], kFloats);
  const int64_t F = gu.cols / 2;
  const Mat q = c.mat(v[1], kCodes, gu.rows, F);
  float* qs = c.need(v[2], gu.rows);
  const float* row = c.f32(v[3], gu.rows);
  const float* col = c.f32(v[4], 2 * F);
  const int act = c.integer(v[5]);
  if (!c.ready() || gu.cols % 2 || F > 16384 || (act != 0 && act != 1)) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("gated_act_quant", [&] {
    return api.gated_act_quant(gu.p, code_of(gu.type), gu.ld, (int)gu.rows, (int)F, row, col, act, q.p, q.ld, qs, s);
  });
}

// res, delta, delta_row, delta_col, bias, gate, write_res, layernorm, weight, beta, mod_scale, mod_shift, q, q_scale, y,
// eps, mod_index
PyObject* residual_norm_quant(PyObject*, Args v, Py_ssize_t nargs) {
  ARITY(17);
  Call c;
  const Mat r = c.mat(v[0], bit(ScalarType::Float) | bit(ScalarType::BFloat16));
  const int64_t M = r.rows, D = r.cols;
  Mat d;
  int splits = 0;
  if (v[1] != Py_None) {
    const at::Tensor* t = c.tensor(v[1]);
    if (!t) Py_RETURN_FALSE;
    if (t->dim() == 3) {  // fp32 partial sums of a K-split GEMM
      if (t->scalar_type() != ScalarType::Float || t->size(0) < 1 || t->size(0) > 8 || t->size(1) != M || t->size(2) != D ||
          !t->is_contiguous())
        Py_RETURN_FALSE;
      splits = (int)t->size(0);
      d.p = t->data_ptr();
      d.ld = D;
    } else {
      d = c.mat(v[1], bit(ScalarType::BFloat16), M, D);
    }
  }
  const float* drow = c.f32(v[2], M);
  const float* dcol = c.f32(v[3], D);
  const float* bias = c.f32(v[4], D);
  const float* gate = c.f32(v[5], D);
  const int write_res = c.flag(v[6]), layernorm = c.flag(v[7]);
  const float* weight = c.f32(v[8], D);
  const float* beta = c.f32(v[9], D);
  const float* ms = c.f32(v[10], D);
  const float* mh = c.f32(v[11], D);
  Mat q, y;
  float* qs = nullptr;
  if (v[12] != Py_None) {
    q = c.mat(v[12], kCodes, M, D);
    qs = c.need(v[13], M);
  } else if (v[13] != Py_None) {
    Py_RETURN_FALSE;
  }
  if (v[14] != Py_None) y = c.mat(v[14], kFloats, M, D);
  const double eps = c.real(v[15]);
  const void* mi = c.vec(v[16], M, ScalarType::Int);
  if (!c.ready() || (ms == nullptr) != (mh == nullptr)) Py_RETURN_FALSE;
  const int y_type = y.p ? code_of(y.type) : IFLB200_F32;
  void* s = c.stream();
  if (splits)
    return finish("residual_norm_quant_partials", [&] {
      return api.residual_norm_quant_partials(r.p, code_of(r.type), r.ld, (int)M, (int)D, static_cast<const float*>(d.p), splits,
                                              d.ld, drow, dcol, bias, gate, write_res, layernorm, weight, beta, ms, mh,
                                              static_cast<const int32_t*>(mi), (float)eps, q.p, q.ld, qs, y.p, y_type, y.ld, s);
    });
  return finish("residual_norm_quant", [&] {
    return api.residual_norm_quant(r.p, code_of(r.type), r.ld, (int)M, (int)D, d.p, d.ld, drow, dcol, bias, gate, write_res,
                                   layernorm, weight, beta, ms, mh, static_cast<const int32_t*>(mi), (float)eps, q.p, q.ld, qs,
                                   y.p, y_type, y.ld, s);
  });
}

// ------------------------------------------------------------------------------------------------
// QKV consumers, attention merge
// ------------------------------------------------------------------------------------------------
struct Heads {
  void* p = nullptr;
  int64_t rows = 0, st = 0, sh = 0;
};
Heads heads_out(Call& c, PyObject* o, int64_t heads, int64_t hd, ScalarType type) {
  Heads h;
  const at::Tensor* t = c.tensor(o);
  if (!t) return h;
  c.ok = t->dim() == 3 && t->scalar_type() == type && t->size(1) == heads && t->size(2) == hd && (hd <= 1 || t->stride(2) == 1);
  if (!c.ok) return h;
  h.p = t->data_ptr();
  h.rows = t->size(0);
  h.st = t->stride(0);
  h.sh = t->stride(1);
  return h;
}

// position table float32 [>= rows, S]
const float* positions(Call& c, PyObject* o, int64_t rows, int64_t* ld) {
  *ld = 0;
  if (o == Py_None) return nullptr;
  const at::Tensor* t = c.tensor(o);
  if (!t) return nullptr;
  c.ok = t->scalar_type() == ScalarType::Float && t->dim() == 2 && (t->size(1) <= 1 || t->stride(1) == 1) && t->size(0) >= rows;
  if (!c.ok) return nullptr;
  *ld = t->stride(0);
  return static_cast<const float*>(t->data_ptr());
}

// qkv, q_out, k_out, v_out, heads_q, heads_kv, head_dim, row, col, bias, inv_freq, pos, sections, q_norm, k_norm, eps, kv_base
PyObject* qkv_split(PyObject*, Args v, Py_ssize_t nargs) {
  ARITY(17);
  Call c;
  const Mat x = c.mat(v[0], kFloats);
  const int hq = c.integer(v[4]), hkv = c.integer(v[5]), hd = c.integer(v[6]);
  if (!c.ok || hq < 0 || hkv < 0 || hd < 2 || hd > 512 || hd % 2 || x.cols != ((int64_t)hq + 2 * (int64_t)hkv) * hd) Py_RETURN_FALSE;
  const at::Tensor* q0 = c.tensor(v[1]);
  if (!q0 || !(kFloats & bit(q0->scalar_type()))) Py_RETURN_FALSE;
  const ScalarType ot = q0->scalar_type();
  const int64_t T = x.rows;
  const Heads q = heads_out(c, v[1], hq, hd, ot), k = heads_out(c, v[2], hkv, hd, ot), w = heads_out(c, v[3], hkv, hd, ot);
  const float* row = c.f32(v[7], T);
  const float* col = c.f32(v[8], x.cols);
  const float* bias = c.f32(v[9], x.cols);
  const float* inv = c.f32(v[10], hd / 2);
  int64_t ld_pos;
  const float* pos = positions(c, v[11], T, &ld_pos);
  const void* sec = c.vec(v[12], hd / 2, ScalarType::Int);
  const float* qn = c.f32(v[13], hd);
  const float* kn = c.f32(v[14], hd);
  const double eps = c.real(v[15]);
  const bool dynamic = THPVariable_Check(v[16]);
  const void* base_dev = dynamic ? c.vec(v[16], 1, ScalarType::Int) : nullptr;
  const int base = dynamic ? 0 : c.integer(v[16]);
  if (!c.ready() || q.rows < T || (inv && !pos) || (qn == nullptr) != (kn == nullptr) ||
      (!dynamic && (base < 0 || base + T > std::min(k.rows, w.rows))))
    Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("qkv_split", [&] {
    return api.qkv_split(x.p, code_of(x.type), T > 1 ? x.ld : x.cols, (int)T, hq, hkv, hd, row, col, bias, qn, kn, (float)eps,
                         inv, pos, ld_pos, static_cast<const int32_t*>(sec), static_cast<const int32_t*>(base_dev), base, q.p,
                         q.st, q.sh, k.p, k.st, k.sh, w.p, w.st, w.sh, code_of(ot), s);
  });
}

struct Pool {
  void* p = nullptr;
  int64_t sb = 0, ss = 0;
};
Pool pool(Call& c, PyObject* o, int64_t D, ScalarType type) {
  Pool r;
  if (o == Py_None) return r;
  const at::Tensor* t = c.tensor(o);
  if (!t) return r;
  c.ok = t->dim() == 3 && t->size(2) == D && (D <= 1 || t->stride(2) == 1) && t->scalar_type() == type;
  if (!c.ok) return r;
  r.p = t->data_ptr();
  r.sb = t->stride(0);
  r.ss = t->stride(1);
  return r;
}

// raw, q_out, heads, head_dim, tokens, k_pool, v_pool, slots, row, col, bias, q_norm, k_norm, pos, sections, inv_freq, eps
PyObject* wan_qkv(PyObject*, Args v, Py_ssize_t nargs) {
  ARITY(17);
  Call c;
  const Mat x = c.mat(v[0], kFloats);
  const int heads = c.integer(v[2]), hd = c.integer(v[3]), tokens = c.integer(v[4]);
  const int64_t D = (int64_t)heads * hd;
  if (!c.ok || heads < 1 || hd < 2 || hd % 2 || hd > 512 || D > 8192 || tokens < 1 || x.rows % tokens) Py_RETURN_FALSE;
  const Mat q = c.mat(v[1], kFloats, x.rows, D);
  const Pool k = pool(c, v[5], D, q.type), w = pool(c, v[6], D, q.type);
  const int parts = 1 + (v[5] != Py_None) + (v[6] != Py_None);
  if (!c.ok || (v[6] != Py_None && v[5] == Py_None) || x.cols < parts * D) Py_RETURN_FALSE;
  const void* slots = c.vec(v[7], tokens, ScalarType::Int);
  const float* row = c.f32(v[8], x.rows);
  const float* col = c.f32(v[9], parts * D);
  const float* bias = c.f32(v[10], parts * D);
  const float* qn = c.f32(v[11], D);
  const float* kn = c.f32(v[12], D);
  int64_t ld_pos;
  const float* pos = positions(c, v[13], tokens, &ld_pos);
  const void* sec = c.vec(v[14], hd / 2, ScalarType::Int);
  const float* inv = c.f32(v[15], hd / 2);
  const double eps = c.real(v[16]);
  if (!c.ready() || (inv && (!pos || !sec))) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("wan_qkv", [&] {
    return api.wan_qkv(x.p, code_of(x.type), x.rows > 1 ? x.ld : x.cols, (int)x.rows, tokens, heads, hd, row, col, bias, qn, kn,
                       (float)eps, inv, pos, ld_pos, static_cast<const int32_t*>(sec), static_cast<const int32_t*>(slots), q.p,
                       x.rows > 1 ? q.ld : D, k.p, k.sb, k.ss, w.p, w.sb, w.ss, code_of(q.type), s);
  });
}

// po, pm, pl, splits, batch, tokens, heads_q, heads_kv, head_dim, out, q8, q8_scale
PyObject* attn_combine(PyObject*, Args v, Py_ssize_t nargs) {
  ARITY(12);
  Call c;
  const int splits = c.integer(v[3]), batch = c.integer(v[4]), tokens = c.integer(v[5]), hq = c.integer(v[6]),
            hkv = c.integer(v[7]), hd = c.integer(v[8]);
  if (!c.ok || splits < 0 || batch < 0 || tokens < 0 || hq < 1 || hkv < 1 || hq % hkv || hd < 4 || hd % 4 || hd > 512 ||
      (int64_t)hq * hd > 8192 || (v[9] == Py_None && v[10] == Py_None))
    Py_RETURN_FALSE;
  int64_t width = 1;
  while (width < hd) width <<= 1;
  const int64_t states = (int64_t)splits * batch * hkv * tokens * (hq / hkv);
  const float* po = c.need(v[0], states * width);
  const float* pm = c.need(v[1], states);
  const float* pl = c.need(v[2], states);
  void* out = nullptr;
  int out_type = IFLB200_F32;
  int64_t so[3] = {0, 0, 0};
  if (v[9] != Py_None) {
    const at::Tensor* t = c.tensor(v[9]);
    if (!t || !(kFloats & bit(t->scalar_type())) || t->dim() != 4 || t->size(0) != batch || t->size(1) != tokens ||
        t->size(2) != hq || t->size(3) != hd || t->stride(3) != 1)
      Py_RETURN_FALSE;
    out = t->data_ptr();
    out_type = code_of(t->scalar_type());
    for (int i = 0; i < 3; ++i) so[i] = t->stride(i);
  }
  Mat q;
  float* qs = nullptr;
  if (v[10] != Py_None) {
    q = c.mat(v[10], kCodes, tokens, (int64_t)hq * hd);
    qs = c.need(v[11], tokens);
    if (batch != 1) Py_RETURN_FALSE;
  }
  if (!c.ready()) Py_RETURN_FALSE;
  void* s = c.stream();
  return finish("attn_combine_quant", [&] {
    return api.attn_combine_quant(po, pm, pl, splits, batch, tokens, hq, hkv, hd, out, out_type, so[0], so[1], so[2], q.p, q.ld,
                                  qs, s);
  });
}

// ------------------------------------------------------------------------------------------------
// Per-tensor pack and the projection module
// ------------------------------------------------------------------------------------------------
const at::Tensor* bf16_input(Call& c, PyObject* o) {
  const at::Tensor* t = c.tensor(o);
  return t && t->scalar_type() == ScalarType::BFloat16 && t->is_contiguous() && t->numel() > 0 ? t : nullptr;
}
at::Tensor empty_on(const at::Tensor& like, at::IntArrayRef size, ScalarType type) {
  return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}

// x -> (codes, scale), or None when x is not the plain case
PyObject* dynamic_pack(PyObject*, Args v, Py_ssize_t nargs) {
  ARITY(1);
  Call c;
  const at::Tensor* x = bf16_input(c, v[0]);
  if (!x || !c.ready()) Py_RETURN_NONE;
  const int64_t n = x->numel();
  at::Tensor codes, scale;
  const int status = unlocked([&] {
    const size_t nbytes = api.pack_workspace_bytes(n);
    codes = empty_on(*x, x->sizes(), ScalarType::Float8_e4m3fn);
    scale = empty_on(*x, {1}, ScalarType::Float);
    const c10::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate(nbytes);
    return api.dynamic_pack_bf16_e4m3(x->data_ptr(), n, codes.data_ptr(), static_cast<float*>(scale.data_ptr()), ws.get(), nbytes,
                                      c.stream());
  });
  if (status != 0) return failed(status, "dynamic_pack_bf16_e4m3");
  PyObject* a = THPVariable_Wrap(std::move(codes));
  PyObject* b = a ? THPVariable_Wrap(std::move(scale)) : nullptr;
  PyObject* pair = b ? PyTuple_Pack(2, a, b) : nullptr;
  Py_XDECREF(a);
  Py_XDECREF(b);
  return pair;
}

// x, weight_fp8 [N, K], weight_scale [1], bias (bf16 [N] or None) -> x @ weight^T [..., N] bf16, or None when the
// arguments are not the plain case.  One scratch allocation holds the codes, their scale and the
// partial maxima; it goes back to the allocator in stream order, like any temporary of the caller's stream.
PyObject* projection(PyObject*, Args v, Py_ssize_t nargs) {
  ARITY(4);
  Call c;
  const at::Tensor* x = bf16_input(c, v[0]);
  const Mat w = c.mat(v[1], kCodes);
  int64_t ns = 0, nb = 0;
  const float* ws = static_cast<float*>(c.vec(v[2], 1, ScalarType::Float, &ns));
  const void* bias = c.vec(v[3], w.rows, ScalarType::BFloat16, &nb);
  if (!x || !ws || !c.ready() || x->dim() < 1 || x->size(-1) != w.cols || ns != 1 || w.cols % 16 || w.rows % 16 ||
      (bias && nb != w.rows))
    Py_RETURN_NONE;
  const int64_t n = x->numel(), K = w.cols, N = w.rows, M = n / K;
  if (M > INT32_MAX) Py_RETURN_NONE;
  const char* what = "dynamic_pack_bf16_e4m3";
  at::Tensor out;
  const int status = unlocked([&] {
    c10::SmallVector<int64_t, 8> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = N;
    out = empty_on(*x, shape, ScalarType::BFloat16);
    const size_t nbytes = api.pack_workspace_bytes(n);
    const int64_t at_scale = (n + 255) / 256 * 256, at_partials = at_scale + 256;
    const c10::DataPtr scratch = c10::cuda::CUDACachingAllocator::get()->allocate(at_partials + nbytes);
    char* codes = static_cast<char*>(scratch.get());
    float* scale = reinterpret_cast<float*>(codes + at_scale);
    void* s = c.stream();
    const int packed = api.dynamic_pack_bf16_e4m3(x->data_ptr(), n, codes, scale, codes + at_partials, nbytes, s);
    if (packed != 0) return packed;
    what = "fp8_linear";
    return api.fp8_linear(codes, K, w.p, w.ld, (int)M, (int)N, (int)K, scale, M != 1 ? 0 : 1, ws, 0, bias, IFLB200_BF16,
                          IFLB200_ROUND_EXACT, out.data_ptr(), IFLB200_BF16, N, s);
  });
  if (status != 0) return failed(status, what);
  return THPVariable_Wrap(std::move(out));
}

// ------------------------------------------------------------------------------------------------
PyObject* bind(PyObject*, PyObject* table) {  // {"iflb200_...": address}
  Api next;
  if (!PyDict_Check(table)) {
    PyErr_SetString(PyExc_TypeError, "bind takes a dict of entry-point addresses");
    return nullptr;
  }
#define IFLB200_BIND(name)                                                                                  \
  {                                                                                                         \
    PyObject* o = PyDict_GetItemString(table, "iflb200_" #name);                                            \
    void* p = o ? PyLong_AsVoidPtr(o) : nullptr;                                                            \
    if (!p) {                                                                                               \
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, "no address for iflb200_" #name);              \
      return nullptr;                                                                                       \
    }                                                                                                       \
    next.name = reinterpret_cast<decltype(next.name)>(p);                                                   \
  }
  IFLB200_CALLS(IFLB200_BIND)
#undef IFLB200_BIND
  next.bound = true;
  api = next;
  Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, Args, Py_ssize_t)>
PyObject* guarded(PyObject* self, Args v, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, v, n);
  END_HANDLE_TH_ERRORS
}

#define METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&guarded<f>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    METHOD(gemm), METHOD(fp8_linear), METHOD(fp8_linear_residual), METHOD(fp8_linear_gated), METHOD(gemm_partials),
    METHOD(row_quant), METHOD(quant_from_amax), METHOD(dequant_rows), METHOD(gated_act_quant), METHOD(residual_norm_quant),
    METHOD(qkv_split), METHOD(wan_qkv), METHOD(attn_combine), METHOD(dynamic_pack), METHOD(projection),
    {"bind", bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", "Calls from tensors to libiflb200.so", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// `torch_version`: whose tensors this file was compiled for; the loader binds it under that torch only
PyMODINIT_FUNC PyInit__calls() {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) Py_CLEAR(m);
  return m;
}
