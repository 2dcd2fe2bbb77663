// Host side of the operator layer (ops.py) as a CPython extension: argument checks, output allocation, the current stream
// and the call into the C-ABI (libkf_b200.so) in one native call per operator.
//
// What bounds it: a small model called eagerly is a hundred launches of 3 to 10 us each, and the same steps in Python
// (attribute and dict look-ups, a ctypes structure of 30 fields, a stream object, a closure) took 12 to 16 us per operator.
// Here an operator costs its launch (about 2 us), one allocation where it returns a new tensor and about 1 us for the rest.
//
// Containers are the Python ones: an operand is any object with the attributes M, K, fmt, q, sf, ts (ops.ActBuf), a weight any
// object with N, K, fmt, q, sf, ts and optionally settled (ops.QWeight).  Errors are KfError of the package.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdarg>

#include "../../../include/kf_b200.h"

namespace {

PyObject* g_error = nullptr;                                   // KfError
PyObject *s_M, *s_N, *s_K, *s_fmt, *s_q, *s_sf, *s_ts, *s_settled;         // interned attribute names
PyObject* g_fmt_names[4];                                      // interned "mx8", "nv4", "mx4", "bf16": index = KF_FMT_*

struct Failed {};                                              // a Python exception is set

[[noreturn]] void fail(const char* format, ...) {
  va_list ap;
  va_start(ap, format);
  PyErr_FormatV(g_error, format, ap);
  va_end(ap);
  throw Failed{};
}

void need(bool cond, const char* what) {
  if (!cond) fail("%s", what);
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) fail("%s must be a tensor", what);
  return THPVariable_Unpack(o);
}

const char* const NO_CPU = "operands must live on a CUDA device (there is no CPU path)";

const at::Tensor& cuda_tensor(PyObject* o, const char* what) {
  const at::Tensor& t = tensor(o, what);
  if (!t.is_cuda()) fail("%s", NO_CPU);
  return t;
}

[[noreturn]] void divides_by_zero(const char* what) {          // what Python arithmetic on the shapes raises
  PyErr_SetString(PyExc_ZeroDivisionError, what);
  throw Failed{};
}

// rows of x seen as [rows, d]
int64_t rows_of(const at::Tensor& x, int64_t d, const char* what) {
  if (d == 0) divides_by_zero(what);
  return x.numel() / d;
}

at::Tensor opt_tensor(PyObject* o, const char* what) { return o == Py_None ? at::Tensor() : cuda_tensor(o, what); }
// pointer of an optional CUDA tensor (None = null)
void* opt_ptr(PyObject* o, const char* what) { return o == Py_None ? nullptr : cuda_tensor(o, what).data_ptr(); }

// An owned reference: an attribute may be a property, whose value nobody else holds.
class Ref {
 public:
  explicit Ref(PyObject* p) : p_(p) {}
  Ref(Ref&& o) noexcept : p_(o.p_) { o.p_ = nullptr; }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p_); }
  operator PyObject*() const { return p_; }

 private:
  PyObject* p_;
};

Ref attr(PyObject* o, PyObject* name) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (!v) throw Failed{};
  return Ref(v);
}

int64_t to_int(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Failed{};
  return v;
}

double to_float(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Failed{};
  return v;
}

bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw Failed{};
  return v != 0;
}

int fmt_code(PyObject* name) {
  for (int i = 0; i < 4; ++i)
    if (name == g_fmt_names[i]) return i;
  if (PyUnicode_Check(name))
    for (int i = 0; i < 4; ++i)
      if (PyUnicode_Compare(name, g_fmt_names[i]) == 0) return i;
  fail("unknown operand format %R", name);
}

struct Operand {                                               // ActBuf or QWeight; holds its tensors until the launch is made
  int fmt;
  int64_t rows, K;
  at::Tensor q, sf, ts;                                        // sf: undefined for bf16, ts: undefined unless nv4
  void *pq, *psf, *pts;
};

Operand operand(PyObject* o, PyObject* rows_attr, const char* what) {
  Operand r;
  r.rows = to_int(attr(o, rows_attr));
  r.K = to_int(attr(o, s_K));
  r.fmt = fmt_code(attr(o, s_fmt));
  r.q = cuda_tensor(attr(o, s_q), what);
  r.pq = r.q.data_ptr();
  r.sf = opt_tensor(attr(o, s_sf), what);
  r.psf = r.sf.defined() ? r.sf.data_ptr() : nullptr;
  r.ts = opt_tensor(attr(o, s_ts), what);
  r.pts = r.ts.defined() ? r.ts.data_ptr() : nullptr;
  return r;
}
Operand act(PyObject* o, const char* what) { return operand(o, s_M, what); }
Operand weight(PyObject* o) { return operand(o, s_N, "weight"); }

int dtype_code(at::ScalarType t) { return t == at::kFloat ? KF_F32 : t == at::kBFloat16 ? KF_BF16 : t == at::kHalf ? KF_F16 : -1; }
at::ScalarType dtype_of(int code) { return code == KF_F32 ? at::kFloat : code == KF_BF16 ? at::kBFloat16 : at::kHalf; }

// fp32, contiguous, n elements; None passes
const float* f32_vec(PyObject* o, int64_t n, const char* what) {
  if (o == Py_None) return nullptr;
  const at::Tensor& t = tensor(o, what);
  if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.numel() != n) fail("gemm: %s must be contiguous fp32 with %lld elements", what, (long long)n);
  if (!t.is_cuda()) fail("%s", NO_CPU);
  return t.data_ptr<float>();
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

void check(int status, const char* what) {
  if (status != 0) fail("%s failed with status %d: %s", what, status, kf_last_error_string());
}

// Other threads run while this one is inside an allocation or the library: a launch blocks when the stream's queue is full.
class Unlocked {
 public:
  Unlocked() : state_(PyEval_SaveThread()) {}
  Unlocked(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state_); }

 private:
  PyThreadState* state_;
};

// fn(args...) of the C-ABI without the interpreter lock; the arguments have been worked out with it
template <typename... P, typename... A>
void launch(const char* what, int (*fn)(P...), A... args) {
  int status;
  {
    const Unlocked unlocked;
    status = fn(args...);
  }
  check(status, what);
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, at::Device device) {
  const Unlocked unlocked;
  return at::Tensor(at::detail::empty_cuda(sizes, dtype, device, std::nullopt));
}

PyObject* new_ref(PyObject* o) {
  Py_INCREF(o);
  return o;
}

PyObject* pair(at::Tensor a, at::Tensor b) {
  PyObject *x = THPVariable_Wrap(std::move(a)), *y = THPVariable_Wrap(std::move(b));
  PyObject* t = PyTuple_New(2);
  PyTuple_SET_ITEM(t, 0, x);
  PyTuple_SET_ITEM(t, 1, y);
  return t;
}

// ------------------------------------------------------------------------------------------------ GEMM
// KF_G_W_STATIC lets the kernel read weights before the wait that makes the predecessor's writes visible, so it is claimed only for
// weights whose writes the host has seen complete and that nothing has written since: `settled` is (q, sf, sum of their version counters)
// at that moment (ops.settled), None where the host did not wait.  torch counts its in-place writes, writable() those of the operators
// here; other tensors in the place of those two, or an object without the attribute, claim nothing.  bmm_nt takes activations and does
// not claim it either.
bool weight_settled(PyObject* o, const at::Tensor& q, const at::Tensor& sf) {
  PyObject* p = PyObject_GetAttr(o, s_settled);
  if (!p) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw Failed{};
    PyErr_Clear();
    return false;
  }
  const Ref seen(p);
  if (!PyTuple_Check(p) || PyTuple_GET_SIZE(p) != 3) return false;
  auto same = [&](Py_ssize_t i, const at::Tensor& t) {
    PyObject* held = PyTuple_GET_ITEM(p, i);
    return t.defined() ? THPVariable_Check(held) && THPVariable_Unpack(held).is_same(t) : held == Py_None;
  };
  if (!same(0, q) || !same(1, sf) || q.is_inference() || (sf.defined() && sf.is_inference())) return false;   // an inference tensor has no version counter
  return (int64_t)q._version() + (sf.defined() ? (int64_t)sf._version() : 0) == to_int(PyTuple_GET_ITEM(p, 2));
}
int w_static(PyObject* o, const Operand& W) { return weight_settled(o, W.q, W.sf) ? KF_G_W_STATIC : 0; }

// out is about to be written: counted as torch counts an in-place operation
void writable(const at::Tensor& out) {
  if (!out.is_inference()) out.unsafeGetTensorImpl()->bump_version();
}
void writable(const Operand& out) {
  writable(out.q);
  if (out.sf.defined()) writable(out.sf);
}
// A side, W side and the common fields; returns M
int64_t gemm_fill(kf_gemm_params& p, PyObject* a, const Operand& W, int epi) {
  int64_t M;
  if (THPVariable_Check(a)) {
    const at::Tensor& t = THPVariable_Unpack(a);
    if (W.fmt != KF_FMT_BF16 || t.scalar_type() != at::kBFloat16 || t.dim() != 2 || !t.is_contiguous() || t.size(1) != W.K)
      fail("gemm: a plain tensor operand must be contiguous bf16 [M, K] with a bf16 weight");
    if (!t.is_cuda()) fail("%s", NO_CPU);
    M = t.size(0);
    p.A = t.data_ptr();
  } else {
    const Operand A = act(a, "gemm operand");
    if (A.fmt != W.fmt || A.K != W.K) fail("gemm: operand mismatch A %U K=%lld vs W %U K=%lld", g_fmt_names[A.fmt], (long long)A.K, g_fmt_names[W.fmt], (long long)W.K);
    M = A.rows;
    p.A = A.pq;
    p.SFA = A.psf;
    p.ts_a = static_cast<const float*>(A.pts);
  }
  p.fmt = W.fmt;
  p.epi = epi;
  p.M = (int)M;
  p.N = (int)W.rows;
  p.K = (int)W.K;
  p.W = W.pq;
  p.SFW = W.psf;
  p.ts_w = static_cast<const float*>(W.pts);
  return M;
}

void gemm_run(const kf_gemm_params& p, const char* what) { launch(what, kf_gemm_bs, &p, stream()); }

// a, W, bias, out | None, out dtype code, flags
PyObject* gemm_plain(PyObject* const* v) {
  const Operand W = weight(v[1]);
  kf_gemm_params p = {};
  const float* bias = f32_vec(v[2], W.rows, "bias");
  const int64_t M = gemm_fill(p, v[0], W, KF_EPI_PLAIN);
  p.bias = bias;
  p.flags = (int)to_int(v[5]) | w_static(v[1], W);
  if (v[3] == Py_None) {
    p.out_dtype = (int)to_int(v[4]);
    at::Tensor out = empty({M, W.rows}, dtype_of(p.out_dtype), W.q.device());
    p.C = out.data_ptr();
    gemm_run(p, "gemm_plain");
    return THPVariable_Wrap(std::move(out));
  }
  const at::Tensor& out = cuda_tensor(v[3], "out");
  p.out_dtype = dtype_code(out.scalar_type());
  p.C = out.data_ptr();
  writable(out);
  gemm_run(p, "gemm_plain");
  return new_ref(v[3]);
}

// (group, stride, offset) as any iterable of three integers
struct RowMap {
  int group, stride, offset;
};
RowMap row_map(PyObject* o) {
  PyObject* seq = PySequence_Fast(o, "gemm_res: row_map must be (group, stride, offset)");
  if (!seq) throw Failed{};
  int value[3] = {0, 0, 0};
  bool ok = PySequence_Fast_GET_SIZE(seq) == 3;
  if (!ok) PyErr_Format(PyExc_ValueError, "gemm_res: row_map must be (group, stride, offset), got %zd values", PySequence_Fast_GET_SIZE(seq));
  for (int i = 0; ok && i < 3; ++i) {
    const long n = PyLong_AsLong(PySequence_Fast_GET_ITEM(seq, i));
    ok = !(n == -1 && PyErr_Occurred());
    if (ok && n != (int)n) {
      PyErr_Format(PyExc_OverflowError, "gemm_res: row_map value %ld does not fit a 32-bit integer", n);
      ok = false;
    }
    value[i] = (int)n;
  }
  Py_DECREF(seq);
  if (!ok) throw Failed{};
  if (value[0] == 0) divides_by_zero("gemm_res: row_map with a group of 0 rows");
  return {value[0], value[1], value[2]};
}

// a, W, bias, gamma, res, out | None, row_map | None
PyObject* gemm_res(PyObject* const* v) {
  const Operand W = weight(v[1]);
  kf_gemm_params p = {};
  const float* bias = f32_vec(v[2], W.rows, "bias");
  const float* gamma = f32_vec(v[3], W.rows, "gamma");
  const int64_t M = gemm_fill(p, v[0], W, KF_EPI_RES);
  p.bias = bias;
  p.gamma = gamma;
  p.flags = w_static(v[1], W);
  p.R = f32_vec(v[4], M * W.rows, "res");
  p.out_dtype = KF_F32;
  if (v[5] == Py_None) {
    if (v[6] != Py_None) fail("gemm_res: a row mapping needs the output tensor");
    const at::Tensor& res = tensor(v[4], "res");
    at::Tensor out = [&] {
      const Unlocked unlocked;
      return at::empty_like(res);
    }();
    p.C = out.data_ptr();
    gemm_run(p, "gemm_res");
    return THPVariable_Wrap(std::move(out));
  }
  const at::Tensor& out = cuda_tensor(v[5], "out");
  need(out.scalar_type() == at::kFloat && out.is_contiguous(), "gemm_res: out must be contiguous fp32");
  if (v[6] != Py_None) {
    const RowMap m = row_map(v[6]);
    if (M % m.group || out.numel() != (M / m.group) * m.stride * W.rows || (int64_t)m.offset + m.group > m.stride)
      fail("gemm_res: row mapping (%d, %d, %d) does not fit M=%lld rows into an output of %lld values", m.group, m.stride, m.offset, (long long)M, (long long)out.numel());
    p.out_row_group = m.group;
    p.out_row_stride = m.stride;
    p.out_row_offset = m.offset;
  }
  p.C = out.data_ptr();
  writable(out);
  gemm_run(p, "gemm_res");
  return new_ref(v[5]);
}

// a, W, bias, sin, cos, Ntok, prefix, H, out dtype code, flags
PyObject* qkv_rope(PyObject* const* v) {
  const Operand W = weight(v[1]);
  kf_gemm_params p = {};
  const float* bias = f32_vec(v[2], W.rows, "bias");
  const at::Tensor &sin = tensor(v[3], "sin"), &cos = tensor(v[4], "cos");
  const int64_t Ntok = to_int(v[5]), prefix = to_int(v[6]), H = to_int(v[7]);
  need(sin.scalar_type() == at::kFloat && cos.scalar_type() == at::kFloat && sin.is_contiguous() && cos.is_contiguous() && sin.dim() > 0 && sin.size(-1) == 64 &&
           sin.size(0) >= Ntok - prefix && cos.sizes() == sin.sizes(),
       "qkv_rope: sin / cos must be contiguous fp32 [>= Ntok - prefix, 64]");
  need(sin.is_cuda() && cos.is_cuda(), NO_CPU);
  const int64_t M = gemm_fill(p, v[0], W, KF_EPI_ROPE);
  need(Ntok > 0 && M % Ntok == 0, "qkv_rope: M must be a multiple of Ntok");
  p.bias = bias;
  p.sin = sin.data_ptr<float>();
  p.cos = cos.data_ptr<float>();
  p.Ntok = (int)Ntok;
  p.prefix = (int)prefix;
  p.H = (int)H;
  p.out_dtype = (int)to_int(v[8]);
  p.flags = (int)to_int(v[9]) | w_static(v[1], W);
  at::Tensor out = empty({3, M / Ntok, Ntok, H, 64}, dtype_of(p.out_dtype), W.q.device());
  p.C = out.data_ptr();
  gemm_run(p, "qkv_rope");
  return THPVariable_Wrap(std::move(out));
}

// a, W, bias, out (ActBuf), flags, y_dbg | None
PyObject* gemm_gelu_q(PyObject* const* v) {
  const Operand W = weight(v[1]);
  kf_gemm_params p = {};
  const float* bias = f32_vec(v[2], W.rows, "bias");
  const int64_t M = gemm_fill(p, v[0], W, KF_EPI_QUANT);
  const Operand out = act(v[3], "out");
  if (out.rows != M || out.K != W.rows)
    fail("gemm_gelu_q: out must be [%lld, %lld], got [%lld, %lld]", (long long)M, (long long)W.rows, (long long)out.rows, (long long)out.K);
  p.bias = bias;
  p.y_dbg = const_cast<float*>(f32_vec(v[5], M * W.rows, "y_dbg"));
  p.out_dtype = KF_BF16;
  p.out_fmt = out.fmt;
  p.Qo = out.pq;
  p.SFo = out.psf;
  p.tso = static_cast<const float*>(out.pts);
  p.flags = (int)to_int(v[4]) | w_static(v[1], W);
  writable(out);
  gemm_run(p, "gemm_gelu_q");
  return new_ref(v[3]);
}

// a [B, Q, K], w [B, P, K], out | None
PyObject* bmm_nt(PyObject* const* v) {
  const at::Tensor &a = cuda_tensor(v[0], "a"), &w = cuda_tensor(v[1], "w");
  need(a.dim() == 3 && w.dim() == 3 && a.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && a.is_contiguous() && w.is_contiguous() &&
           a.size(0) == w.size(0) && a.size(2) == w.size(2),
       "bmm_nt: a [B, Q, K] and w [B, P, K] must be contiguous bf16 with equal B and K");
  const int64_t B = a.size(0), Q = a.size(1), K = a.size(2), P = w.size(1);
  at::Tensor out;
  if (v[2] == Py_None) {
    out = empty({B, Q, P}, at::kBFloat16, a.device());
  } else {
    out = cuda_tensor(v[2], "out");
    if (out.dim() != 3 || out.size(0) != B || out.size(1) != Q || out.size(2) != P || out.scalar_type() != at::kBFloat16 || !out.is_contiguous())
      fail("bmm_nt: out must be contiguous bf16 [%lld, %lld, %lld]", (long long)B, (long long)Q, (long long)P);
    writable(out);
  }
  kf_gemm_params p = {};
  p.fmt = KF_FMT_BF16;
  p.epi = KF_EPI_PLAIN;
  p.M = (int)(B * Q);
  p.N = (int)P;
  p.K = (int)K;
  p.A = a.data_ptr();
  p.W = w.data_ptr();
  p.C = out.data_ptr();
  p.out_dtype = KF_BF16;
  p.batch = (int)B;
  p.a_rows_per_batch = (int)Q;
  p.w_rows_per_batch = (int)P;
  gemm_run(p, "bmm_nt");
  return v[2] == Py_None ? THPVariable_Wrap(std::move(out)) : new_ref(v[2]);
}

// a, W, bias, out, rows per image, tokens per image, row offset, flags
PyObject* gemm_tokens(PyObject* const* v) {
  const at::Tensor &a = cuda_tensor(v[0], "a"), &out = cuda_tensor(v[3], "out");
  const Operand W = weight(v[1]);
  need(out.scalar_type() == at::kFloat && out.is_contiguous(), "gemm_tokens: out must be contiguous fp32");
  kf_gemm_params p = {};
  p.fmt = KF_FMT_BF16;
  p.epi = KF_EPI_PLAIN;
  p.M = (int)a.size(0);
  p.N = (int)W.rows;
  p.K = (int)W.K;
  p.A = a.data_ptr();
  p.W = W.pq;
  p.bias = static_cast<const float*>(opt_ptr(v[2], "bias"));
  p.C = out.data_ptr();
  p.out_dtype = KF_F32;
  p.out_row_group = (int)to_int(v[4]);
  p.out_row_stride = (int)to_int(v[5]);
  p.out_row_offset = (int)to_int(v[6]);
  p.flags = (int)to_int(v[7]) | w_static(v[1], W);
  writable(out);
  gemm_run(p, "gemm_tokens");
  return new_ref(v[3]);
}

// ------------------------------------------------------------------------------------------------ quantisers and LayerNorm
// x, out, bias, flags
PyObject* quant_rows(PyObject* const* v) {
  const at::Tensor& x = cuda_tensor(v[0], "x");
  const Operand out = act(v[1], "out");
  if (x.dim() != 2 || x.stride(1) != 1 || x.size(0) != out.rows || x.size(1) != out.K) {
    if (x.dim() == 2)
      fail("quant_rows: x must be [M=%lld, K=%lld] with a contiguous last dim, got (%lld, %lld)", (long long)out.rows, (long long)out.K, (long long)x.size(0), (long long)x.size(1));
    fail("quant_rows: x must be [M=%lld, K=%lld] with a contiguous last dim, got %lld dimensions", (long long)out.rows, (long long)out.K, (long long)x.dim());
  }
  const int dt = dtype_code(x.scalar_type());
  if (dt < 0) fail("quant_rows: unsupported dtype %s", c10::toString(x.scalar_type()));
  writable(out);
  launch("quant_rows", kf_quant_rows, out.fmt, dt, x.data_ptr(), x.stride(0), (int)out.rows, (int)out.K, static_cast<const float*>(out.pts),
         static_cast<const float*>(opt_ptr(v[2], "bias")), (int)to_int(v[3]), out.pq, out.psf, stream());
  return new_ref(v[1]);
}

// x, w, b, eps, out, flags, y_dbg
PyObject* ln_quant(PyObject* const* v) {
  const at::Tensor& x = cuda_tensor(v[0], "x");
  const Operand out = act(v[4], "out");
  const int64_t d = x.dim() > 0 ? x.size(-1) : 0, M = d > 0 ? x.numel() / d : 0;
  const bool bf16 = x.scalar_type() == at::kBFloat16;
  if ((x.scalar_type() != at::kFloat && !bf16) || !x.is_contiguous() || M != out.rows || d != out.K)
    fail("ln_quant: x must be contiguous fp32 or bf16 [M=%lld, d=%lld], got [%lld, %lld] %s", (long long)out.rows, (long long)out.K, (long long)M, (long long)d,
         c10::toString(x.scalar_type()));
  writable(out);
  launch("ln_quant", kf_ln_quant, out.fmt, static_cast<const float*>(x.data_ptr()), static_cast<const float*>(opt_ptr(v[1], "w")), static_cast<const float*>(opt_ptr(v[2], "b")),
         (float)to_float(v[3]), (int)M, (int)d, static_cast<const float*>(out.pts), (int)to_int(v[5]) | (bf16 ? KF_Q_IN_BF16 : 0), out.pq, out.psf,
         static_cast<float*>(opt_ptr(v[6], "y_dbg")), stream());
  return new_ref(v[4]);
}

// ts [1] fp32 and ws (two 32-bit words, zero before the first use)
float* scale_target(PyObject* ts, PyObject* ws, void** words) {
  const at::Tensor &t = cuda_tensor(ts, "ts"), &w = cuda_tensor(ws, "ws");
  need(t.scalar_type() == at::kFloat && t.numel() == 1 && w.scalar_type() == at::kInt && w.numel() >= 2 && w.is_contiguous(),
       "amax_scale: ts must be fp32 [1] and ws contiguous int32 [2]");
  *words = w.data_ptr();
  return t.data_ptr<float>();
}

// x, flags, factor, ts, ws
PyObject* amax_scale(PyObject* const* v) {
  const at::Tensor& x = cuda_tensor(v[0], "x");
  const int dt = dtype_code(x.scalar_type());
  need(x.dim() == 2 && x.stride(1) == 1 && dt >= 0, "amax_scale: x must be f32 | bf16 | f16 [M, K] with a contiguous last dim");
  void* ws;
  float* ts = scale_target(v[3], v[4], &ws);
  launch("amax_scale", kf_amax_scale, dt, x.data_ptr(), x.stride(0), (int)x.size(0), (int)x.size(1), (int)to_int(v[1]), (float)to_float(v[2]), ts, ws, stream());
  return new_ref(v[3]);
}

// x, w, b, eps, factor, ts, ws
PyObject* ln_amax_scale(PyObject* const* v) {
  const at::Tensor& x = cuda_tensor(v[0], "x");
  need(x.is_contiguous() && x.dim() > 0 && (x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16), "ln_amax_scale: x must be contiguous fp32 or bf16");
  const int64_t d = x.size(-1), M = rows_of(x, d, "ln_amax_scale: x has a last dimension of 0");
  void* ws;
  float* ts = scale_target(v[5], v[6], &ws);
  launch("ln_amax_scale", kf_ln_amax_scale, dtype_code(x.scalar_type()), x.data_ptr(), static_cast<const float*>(opt_ptr(v[1], "w")), static_cast<const float*>(opt_ptr(v[2], "b")),
         (float)to_float(v[3]), (int)M, (int)d, (float)to_float(v[4]), ts, ws, stream());
  return new_ref(v[5]);
}

// x, w, b, eps, dtype code
PyObject* ln_rows(PyObject* const* v) {
  const at::Tensor& x = cuda_tensor(v[0], "x");
  need(x.scalar_type() == at::kFloat && x.is_contiguous() && x.dim() > 0, "ln_rows: x must be contiguous fp32");
  const int64_t d = x.size(-1), M = rows_of(x, d, "ln_rows: x has a last dimension of 0");
  const int dt = (int)to_int(v[4]);
  at::Tensor y = empty(x.sizes(), dtype_of(dt), x.device());
  launch("ln_rows", kf_ln_rows, x.data_ptr<float>(), static_cast<const float*>(opt_ptr(v[1], "w")), static_cast<const float*>(opt_ptr(v[2], "b")), (float)to_float(v[3]), (int)M, (int)d, dt,
         y.data_ptr(), stream());
  return THPVariable_Wrap(std::move(y));
}

// src, dst, row offset
PyObject* broadcast_rows(PyObject* const* v) {
  const at::Tensor &src = cuda_tensor(v[0], "src"), &dst = cuda_tensor(v[1], "dst");
  need(src.scalar_type() == at::kFloat && dst.scalar_type() == at::kFloat && src.is_contiguous() && dst.is_contiguous() && dst.dim() == 3 && src.dim() > 0 &&
           src.size(-1) == dst.size(2),
       "broadcast_rows: src [R, d] and dst [B, Ntok, d] must be contiguous fp32");
  const int64_t d = dst.size(2), R = rows_of(src, d, "broadcast_rows: src and dst have a last dimension of 0");
  launch("broadcast_rows", kf_broadcast_rows, src.data_ptr<float>(), dst.data_ptr<float>(), (int)R, (int)d, (int)dst.size(0), dst.size(1) * d, to_int(v[2]), stream());
  return new_ref(v[1]);
}

// x, w, b, eps, Q, npre, wcls | None, bcls | None
PyObject* ln_tail(PyObject* const* v) {
  const at::Tensor& x = cuda_tensor(v[0], "x");
  need(x.scalar_type() == at::kFloat && x.is_contiguous() && x.dim() == 3, "ln_tail: x must be contiguous fp32");
  const int64_t B = x.size(0), Ntok = x.size(1), d = x.size(2), Q = to_int(v[4]), npre = to_int(v[5]);
  at::Tensor qb = empty({B * Q, d}, at::kBFloat16, x.device()), xb = empty({B * (Ntok - Q - npre), d}, at::kBFloat16, x.device()), cl;
  int ncls1 = 0;
  const void* wcls = nullptr;
  const float* bcls = nullptr;
  if (v[6] != Py_None) {
    const at::Tensor& wc = cuda_tensor(v[6], "wcls");
    const char* msg = "ln_tail: wcls must be contiguous bf16 [ncls1, d] and bcls fp32 [ncls1]";
    need(wc.scalar_type() == at::kBFloat16 && wc.is_contiguous() && wc.dim() == 2 && wc.size(1) == d && v[7] != Py_None, msg);
    const at::Tensor& bc = cuda_tensor(v[7], "bcls");
    need(bc.scalar_type() == at::kFloat && bc.numel() == wc.size(0), msg);
    ncls1 = (int)wc.size(0);
    wcls = wc.data_ptr();
    bcls = bc.data_ptr<float>();
    cl = empty({B * Q, wc.size(0)}, at::kBFloat16, x.device());
  }
  launch("ln_tail", kf_ln_tail, x.data_ptr<float>(), static_cast<const float*>(opt_ptr(v[1], "w")), static_cast<const float*>(opt_ptr(v[2], "b")), (float)to_float(v[3]), (int)B, (int)Ntok,
         (int)Q, (int)npre, (int)d, qb.data_ptr(), xb.data_ptr(), wcls, bcls, ncls1, ncls1 ? cl.data_ptr() : nullptr, stream());
  if (!ncls1) return pair(std::move(qb), std::move(xb));
  PyObject* t = PyTuple_New(3);
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(qb)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(xb)));
  PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(std::move(cl)));
  return t;
}

// ------------------------------------------------------------------------------------------------ attention
const at::Tensor& qkv_tensor(PyObject* o, const char* msg) {
  const at::Tensor& t = cuda_tensor(o, "qkv");
  need(t.dim() == 5 && t.size(0) == 3 && t.size(4) == 64 && t.is_contiguous() && (t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf), msg);
  return t;
}

// qkv, pre, out | None
PyObject* attn_fwd(PyObject* const* v) {
  const at::Tensor& qkv = qkv_tensor(v[0], "attn_fwd: qkv must be contiguous [3, B, N, H, 64] bf16 or f16");
  const int64_t B = qkv.size(1), N = qkv.size(2), H = qkv.size(3);
  at::Tensor out = v[2] == Py_None ? empty({B, N, H * 64}, qkv.scalar_type(), qkv.device()) : cuda_tensor(v[2], "out");
  if (v[2] != Py_None) writable(out);
  launch("attn_fwd", kf_attn_fwd, dtype_code(qkv.scalar_type()), qkv.data_ptr(), out.data_ptr(), (int)B, (int)N, (int)H, (float)to_float(v[1]), stream());
  return v[2] == Py_None ? THPVariable_Wrap(std::move(out)) : new_ref(v[2]);
}

// qkv, out (ActBuf), pre, flags
PyObject* attn_fwd_quant(PyObject* const* v) {
  const at::Tensor& qkv = qkv_tensor(v[0], "attn_fwd_quant: qkv must be contiguous [3, B, N, H, 64] bf16 or f16");
  const Operand out = act(v[1], "out");
  const int64_t B = qkv.size(1), N = qkv.size(2), H = qkv.size(3);
  if (out.rows != B * N || out.K != H * 64)
    fail("attn_fwd_quant: out must be [%lld, %lld], got [%lld, %lld]", (long long)(B * N), (long long)(H * 64), (long long)out.rows, (long long)out.K);
  writable(out);
  launch("attn_fwd_quant", kf_attn_fwd_quant, dtype_code(qkv.scalar_type()), qkv.data_ptr(), (int)B, (int)N, (int)H, (float)to_float(v[2]), out.fmt, out.pq, out.psf,
         static_cast<const float*>(out.pts), (int)to_int(v[3]), stream());
  return new_ref(v[1]);
}

// ------------------------------------------------------------------------------------------------ patch embed / head / pre / post
// x [B, 3, S, S] bf16
PyObject* im2col_patch16(PyObject* const* v) {
  const at::Tensor& x = cuda_tensor(v[0], "x");
  need(x.scalar_type() == at::kBFloat16 && x.dim() == 4 && x.size(1) == 3 && x.size(2) == x.size(3) && x.is_contiguous(),
       "im2col_patch16: x must be contiguous bf16 [B, 3, S, S]");
  const int64_t B = x.size(0), S = x.size(2), g = S / 16;
  at::Tensor out = empty({B * g * g, 768}, at::kBFloat16, x.device());
  launch("im2col_patch16", kf_im2col_patch16, x.data_ptr(), out.data_ptr(), (int)B, (int)S, stream());
  return THPVariable_Wrap(std::move(out));
}

// g, bias | None, dww, lnw, lnb, B, Hs, Ws, eps, pre_act
PyObject* dw_ln(PyObject* const* v) {
  const at::Tensor &g = cuda_tensor(v[0], "g"), &dww = cuda_tensor(v[2], "dww");
  const int64_t C = g.dim() == 2 ? g.size(1) / 4 : 0, B = to_int(v[5]), Hs = to_int(v[6]), Ws = to_int(v[7]);
  const bool pre = truth(v[9]);
  need(g.scalar_type() == at::kBFloat16 && g.is_contiguous() && g.dim() == 2 && g.size(0) == B * Hs * Ws && dww.dim() == 2 && dww.size(0) == 9 && dww.size(1) == C &&
           (v[1] != Py_None || pre),
       "dw_ln: g must be contiguous bf16 [B*Hs*Ws, 4C] and dww fp32 [9, C]");
  at::Tensor out = empty({B, 2 * Hs, 2 * Ws, C}, at::kBFloat16, g.device());
  launch("dw_ln", kf_dw_ln, g.data_ptr(), static_cast<const float*>(opt_ptr(v[1], "bias")), dww.data_ptr<float>(), static_cast<const float*>(opt_ptr(v[3], "lnw")),
         static_cast<const float*>(opt_ptr(v[4], "lnb")), out.data_ptr(), (int)B, (int)Hs, (int)Ws, (int)C, (float)to_float(v[8]), pre ? 1 : 0, stream());
  return THPVariable_Wrap(std::move(out));
}

// mask_logits, class_logits, want_scores
PyObject* semantic(PyObject* const* v) {
  const at::Tensor &ml = cuda_tensor(v[0], "mask_logits"), &cl = cuda_tensor(v[1], "class_logits");
  need(ml.scalar_type() == at::kBFloat16 && cl.scalar_type() == at::kBFloat16 && ml.is_contiguous() && cl.is_contiguous() && ml.dim() == 4 && cl.dim() > 0,
       "semantic: logits must be contiguous bf16");
  const int64_t B = ml.size(0), Q = ml.size(1), h = ml.size(2), w = ml.size(3), ncls1 = cl.size(-1);
  const bool want = truth(v[2]);
  at::Tensor labels = empty({B, h, w}, at::kByte, ml.device()), scores;
  if (want) scores = empty({B, ncls1, h, w}, at::kFloat, ml.device());
  launch("semantic", kf_semantic, ml.data_ptr(), cl.data_ptr(), (int)B, (int)Q, (int)ncls1 - 1, (int)(h * w), want ? scores.data_ptr<float>() : nullptr, labels.data_ptr<uint8_t>(), stream());
  if (want) return pair(std::move(labels), std::move(scores));
  PyObject* t = PyTuple_New(2);
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(labels)));
  PyTuple_SET_ITEM(t, 1, new_ref(Py_None));
  return t;
}

// a weight: does the next GEMM with it read it ahead of its predecessor's end?
PyObject* reads_weight_early(PyObject* const* v) {
  const Ref q = attr(v[0], s_q), sf = attr(v[0], s_sf);
  return PyBool_FromLong(weight_settled(v[0], tensor(q, "weight"), sf == Py_None ? at::Tensor() : tensor(sf, "weight")));
}

// ------------------------------------------------------------------------------------------------ module
template <PyObject* (*F)(PyObject* const*), int ARGS>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != ARGS) {
    PyErr_Format(PyExc_TypeError, "native operator takes %d arguments, got %zd", ARGS, n);
    return nullptr;
  }
  try {
    return F(args);
  } catch (const Failed&) {
    return nullptr;
  } catch (const c10::OutOfMemoryError& e) {                    // as torch raises it from its own allocations
    PyObject* t = PyImport_ImportModule("torch");
    PyObject* cls = t ? PyObject_GetAttrString(t, "OutOfMemoryError") : nullptr;
    PyErr_SetString(cls ? cls : PyExc_RuntimeError, e.what_without_backtrace());
    Py_XDECREF(cls);
    Py_XDECREF(t);
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

#define KF_ENTRY(f, n) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<f, n>)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {KF_ENTRY(quant_rows, 4),     KF_ENTRY(ln_quant, 7),   KF_ENTRY(ln_rows, 5),  KF_ENTRY(gemm_plain, 6),     KF_ENTRY(gemm_res, 7),
                           KF_ENTRY(qkv_rope, 10),      KF_ENTRY(gemm_gelu_q, 6), KF_ENTRY(bmm_nt, 3),   KF_ENTRY(gemm_tokens, 8),    KF_ENTRY(broadcast_rows, 3),
                           KF_ENTRY(ln_tail, 8),        KF_ENTRY(attn_fwd, 3),   KF_ENTRY(attn_fwd_quant, 4), KF_ENTRY(im2col_patch16, 1), KF_ENTRY(dw_ln, 10),
                           KF_ENTRY(semantic, 3),       KF_ENTRY(amax_scale, 5), KF_ENTRY(ln_amax_scale, 7),
                           KF_ENTRY(reads_weight_early, 1), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_kf_host", "native operator layer over libkf_b200.so", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__kf_host() {
  PyObject* lib = PyImport_ImportModule("lightly_trian_quant_b200._lib");
  if (!lib) return nullptr;
  g_error = PyObject_GetAttrString(lib, "KfError");
  Py_DECREF(lib);
  if (!g_error) return nullptr;
  s_M = PyUnicode_InternFromString("M");
  s_N = PyUnicode_InternFromString("N");
  s_K = PyUnicode_InternFromString("K");
  s_fmt = PyUnicode_InternFromString("fmt");
  s_q = PyUnicode_InternFromString("q");
  s_sf = PyUnicode_InternFromString("sf");
  s_ts = PyUnicode_InternFromString("ts");
  s_settled = PyUnicode_InternFromString("settled");
  const char* names[4] = {"mx8", "nv4", "mx4", "bf16"};
  for (int i = 0; i < 4; ++i) g_fmt_names[i] = PyUnicode_InternFromString(names[i]);
  return PyModule_Create(&g_module);
}
