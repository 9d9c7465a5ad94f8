// The host side of the calls a training step makes most: allocation of the results, checks, launch.  A CPython module
// (mcore_bridge_b200/lib/_mcb200_host.*.so) that takes and returns tensors; the kernels are reached through the C entry points of
// libmcb200.so.  The autograd functions themselves stay in Python (ops/*.py), this is what their bodies did one Python
// call at a time: a GEMM of a small model spent about 24 us in arguments, views and ctypes for 7 us on the device.
//
// Everything runs on the calling thread's current device and stream, with the interpreter's lock held except during a launch.
// A tensor's type, device and size are checked here against what the kernel reads; the first operand's device and the sizes a
// kernel supports are the Python callers' and the C entry points' to check.
#include <Python.h>
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>
#include <initializer_list>

namespace {

using at::Tensor;
typedef long long ll;

// ------------------------------------------------------------------------------------------------ entry points
#define MCB_ENTRIES(X)                                                                                                  \
  X(mcb_gemm_bf16, int, (const void*, ll, ll, ll, int, const void*, ll, ll, ll, int, void*, ll, ll, int, int, int, int, int,  \
                         float, const void*, int, int, const int*, int, int*, int, int, void*))                         \
  X(mcb_rmsnorm_fwd, int, (const void*, const void*, const void*, void*, void*, float*, ll, int, ll, float, int, void*))  \
  X(mcb_rmsnorm_bwd_det, int, (const void*, const void*, const void*, const float*, const void*, void*, void*, int, float*,   \
                               ll, int, ll, float, int, void*))                                                         \
  X(mcb_rmsnorm_bwd_det_y, int, (void*, const void*, const void*, const float*, const void*, void*, void*, int, float*, ll,   \
                                 int, ll, float, int, void*))                                                           \
  X(mcb_rmsnorm_bwd_partial_rows, int, (ll, int))                                                                       \
  X(mcb_glu_fwd, int, (const void*, const float*, void*, ll, int, ll, int, float, float, void*))                        \
  X(mcb_glu_bwd, int, (const void*, const float*, const void*, void*, float*, ll, int, ll, int, float, float, void*))   \
  X(mcb_glu_bwd_act, int, (const void*, const float*, void*, void*, float*, ll, int, ll, int, float, float, void*))     \
  X(mcb_qkv_split_norm_rope_fwd, int, (const void*, const void*, const void*, const float*, const float*, void*, void*, void*,\
                                       void*, ll, int, int, int, int, int, int, int, int, float, ll, void*))            \
  X(mcb_qkv_split_norm_rope_bwd, int, (const void*, const void*, const void*, const float*, const float*, const void*,        \
                                       const void*, const void*, const void*, void*, void*, void*, int, float*, ll, int, int, \
                                       int, int, int, int, int, int, float, ll, void*))                                 \
  X(mcb_qkv_bwd_partial_rows, int, (ll))                                                                                \
  X(mcb_attn_fwd_ranges, int, (const void*, const void*, const void*, const int*, const int*, const float*, void*, float*,    \
                               int, int, int, int, int, float, int*, void*))                                            \
  X(mcb_attn_bwd_ranges, int, (const void*, const void*, const void*, const void*, const void*, const float*, float*, int,    \
                               const int*, const int*, const int*, const int*, void*, void*, void*, int, int, int, int, int,  \
                               float, float*, int, int*, void*))                                                        \
  X(mcb_attn_sink_grad, int, (const float*, const float*, const float*, void*, int, int, int, void*))                   \
  X(mcb_attn_window_starts, int, (const int*, int*, int, int, void*))                                                   \
  X(mcb_sm_count, int, ())

#define MCB_DECLARE(name, ret, args) ret(*name) args = nullptr;
MCB_ENTRIES(MCB_DECLARE)

PyObject* g_kernel_error = nullptr;   // exception class
PyObject* g_make_status = nullptr;    // device index -> address of the device's status words
constexpr int MAX_DEVICES = 64;
int* g_status[MAX_DEVICES] = {nullptr};
ll g_launches = 0;

// ------------------------------------------------------------------------------------------------ helpers
struct Failed {};   // a Python exception is set

void check_count(Py_ssize_t got, Py_ssize_t want, const char* what) {
  if (got == want) return;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, %zd given", what, want, got);
  throw Failed();
}

const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "a tensor is wanted");
    throw Failed();
  }
  return THPVariable_Unpack(o);
}

Tensor optional(PyObject* o) { return o == Py_None ? Tensor() : tensor(o); }

ll integer(PyObject* o) {
  const ll v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Failed();
  return v;
}

float real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Failed();
  return static_cast<float>(v);
}

bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw Failed();
  return v != 0;
}

void require(bool ok, const char* what) {
  if (ok) return;
  PyErr_SetString(PyExc_AssertionError, what);
  throw Failed();
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

int* status_of(const Tensor& t) {
  const int dev = t.get_device();
  require(dev >= 0 && dev < MAX_DEVICES, "device index");
  if (g_status[dev] == nullptr) {
    PyObject* r = PyObject_CallFunction(g_make_status, "i", dev);
    if (r == nullptr) throw Failed();
    void* p = PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    if (p == nullptr) throw Failed();
    g_status[dev] = static_cast<int*>(p);
  }
  return g_status[dev];
}

// One kernel call.  The interpreter's lock is given up meanwhile, as by ctypes: a full launch queue blocks.  An error reads like
// _lib.check_rc's.
template <class... P, class... A>
void launch(const char* what, int (*entry)(P...), A... args) {
  ++g_launches;
  PyThreadState* state = PyEval_SaveThread();
  const int rc = entry(static_cast<P>(args)...);
  PyEval_RestoreThread(state);
  if (rc == 0) return;
  PyErr_Format(g_kernel_error, "%s failed with code %d%s", what, rc, rc > 0 ? " (CUDA error)" : " (bad argument)");
  throw Failed();
}

void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

Tensor rows_of(const Tensor& t, ll width) {           // [rows, width] with a contiguous last dimension
  Tensor r = t.dim() == 2 ? t : t.reshape({-1, width});
  return r.stride(-1) == 1 ? r : r.contiguous();
}

Tensor tma_rows(const Tensor& t) {                    // ... whose rows TMA can address
  Tensor r = t.dim() == 2 ? t : t.reshape({-1, t.size(-1)});
  if (r.stride(1) != 1 || r.stride(0) % 8 != 0 || reinterpret_cast<uintptr_t>(r.data_ptr()) % 16 != 0) r = r.contiguous();
  return r;
}

PyObject* tuple(std::initializer_list<Tensor> ts) {
  PyObject* r = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  if (r == nullptr) throw Failed();
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) {
    PyObject* o = t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None);
    if (o == nullptr) {
      Py_DECREF(r);
      throw Failed();
    }
    PyTuple_SET_ITEM(r, i++, o);
  }
  return r;
}

// An operand a kernel reads at least n elements of one type from, beside `like`; an undefined one is left out.
void operand(const Tensor& t, at::ScalarType type, ll n, const Tensor& like, const char* what) {
  require(!t.defined() || (t.scalar_type() == type && t.numel() >= n && t.device() == like.device()), what);
}

// What a kernel reads one int32 of per query or key from.
Tensor per_token(const Tensor& t, ll n, const Tensor& like, const char* what) {
  operand(t, at::kInt, n, like, what);
  return t.defined() ? t.contiguous() : t;
}

enum Layout { NT = 0, NN = 1, TN = 2 };

// c = op(a) . op(b): NT a [M, K], b [N, K]; NN a [M, K], b [K, N]; TN a [K, M], b [K, N]
Tensor gemm(int layout, const Tensor& a_, const Tensor& b_, const Tensor& bias_, const Tensor& out, bool fp32, bool accumulate,
            float alpha, int max_sms, int force_bn) {
  const Tensor a = tma_rows(a_), b = tma_rows(b_);
  const bool a_mn = layout == TN, b_mn = layout != NT;
  const ll M = a.size(a_mn ? 1 : 0), K = a.size(a_mn ? 0 : 1), N = b.size(b_mn ? 1 : 0);
  require(b.size(b_mn ? 0 : 1) == K, "GEMM operands whose contraction sizes differ");
  require(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && b.device() == a.device(),
          "GEMM operands: bf16 on one device");
  require(!out.defined() || ((out.scalar_type() == at::kFloat || out.scalar_type() == at::kBFloat16) && out.device() == a.device()),
          "GEMM output: bf16 or fp32 on the operands' device");
  require(!out.defined() || layout != TN || out.dim() == 2, "GEMM output of another shape");
  require(!bias_.defined() || (bias_.numel() == N && bias_.device() == a.device()), "GEMM bias: one for every column");
  Tensor c;
  if (out.defined()) {
    c = layout == TN || (out.dim() == 2 && out.size(0) == M && out.size(1) == N) ? out : out.view({M, N});
    require(c.size(0) == M && c.size(1) == N && c.stride(1) == 1, "GEMM output of another shape");
  } else {
    require(!accumulate, "accumulate needs an output tensor");
    c = at::empty({M, N}, a.options().dtype(fp32 ? at::kFloat : at::kBFloat16));
  }
  Tensor bias = bias_;
  if (bias.defined()) bias = bias.to(at::kBFloat16).contiguous();
  launch("mcb_gemm_bf16", mcb_gemm_bf16, a.data_ptr(), a.size(1), a.size(0), a.stride(0), a_mn, b.data_ptr(), b.size(1),
         b.size(0), b.stride(0), b_mn, c.data_ptr(), c.stride(0), 0, c.scalar_type() == at::kFloat, accumulate, M, N, K,
         alpha, ptr(bias), 0, 0, nullptr, 0, status_of(a), max_sms, force_bn, stream());
  return c;
}

void norm_fwd(const Tensor& x2, const Tensor& w, float eps, bool zc, Tensor& y, Tensor& rstd) {
  const ll rows = x2.size(0), H = x2.size(1);
  operand(x2, at::kBFloat16, 0, x2, "norm input: bf16");
  operand(w, at::kBFloat16, H, x2, "norm weight: bf16, one for every column");
  y = at::empty({rows, H}, x2.options());
  rstd = at::empty({rows}, x2.options().dtype(at::kFloat));
  launch("mcb_rmsnorm_fwd", mcb_rmsnorm_fwd, x2.data_ptr(), nullptr, w.data_ptr(), y.data_ptr(), nullptr, rstd.data_ptr(),
         rows, H, x2.stride(0), eps, zc, stream());
}

// `over` replaces dy with the norm's result
void norm_bwd(const Tensor& dy, const Tensor& x2, const Tensor& w, const Tensor& rstd, float eps, bool zc, bool over,
              bool need_dw, Tensor& dx, Tensor& dw) {
  const ll rows = x2.size(0), H = x2.size(1);
  operand(dy, at::kBFloat16, rows * H, x2, "norm gradient: bf16 of the input's size");
  operand(w, at::kBFloat16, H, x2, "norm weight: bf16, one for every column");
  operand(rstd, at::kFloat, rows, x2, "norm: an fp32 for every row");
  dx = at::empty({rows, H}, x2.options());
  Tensor part;
  if (need_dw) {
    dw = rows ? at::empty({H}, w.options()) : at::zeros({H}, w.options());
    part = at::empty({mcb_rmsnorm_bwd_partial_rows(rows, static_cast<int>(H)), H}, x2.options().dtype(at::kFloat));
  }
  if (over)
    launch("mcb_rmsnorm_bwd_det", mcb_rmsnorm_bwd_det_y, dy.data_ptr(), x2.data_ptr(), w.data_ptr(), rstd.data_ptr(), nullptr,
           dx.data_ptr(), ptr(dw), 1, ptr(part), rows, H, x2.stride(0), eps, zc, stream());
  else
    launch("mcb_rmsnorm_bwd_det", mcb_rmsnorm_bwd_det, dy.data_ptr(), x2.data_ptr(), w.data_ptr(), rstd.data_ptr(), nullptr,
           dx.data_ptr(), ptr(dw), 1, ptr(part), rows, H, x2.stride(0), eps, zc, stream());
}

// How many CTAs share one (key tile, kv head) pair in the dK/dV kernel: the smallest divisor of the GQA ratio that puts about three
// CTAs on every SM, or the largest there is; a step of more than twice is taken only while SMs are idle.  dK/dV and the sum of
// the parts, us, whole / in 3, 3, 5 and 3 parts: 3000 tokens, 9 / 3 heads of 128 133 / 63, 8192 in seven sequences, 3 / 1 heads of 64
// 107 / 48, 777, 5 / 1 of 128 35 / 18; 4096, 24 / 8 of 64 171 / 194 (256 pairs).
// MCB200_ATTN_DKV_SPLITS overrides it.
int dkv_splits(ll T, int nq, int nkv) {
  require(nkv > 0, "attention without key heads");
  const int qpg = nq / nkv;
  const char* env = std::getenv("MCB200_ATTN_DKV_SPLITS");
  if (env && *env) {
    char* end;
    const long s = std::strtol(env, &end, 10);
    if (*end) {
      PyErr_Format(PyExc_ValueError, "MCB200_ATTN_DKV_SPLITS is not a number: %s", env);
      throw Failed();
    }
    return s >= 1 && qpg % s == 0 ? static_cast<int>(s) : 1;
  }
  const ll ctas = (T + 127) / 128 * nkv;
  int s = 1;
  for (int next = 2; next <= qpg; ++next)
    if (qpg % next == 0) {
      if (ctas * s >= (next <= 2 * s ? 3ll : 1ll) * mcb_sm_count()) break;
      s = next;
    }
  return s;
}

// ------------------------------------------------------------------------------------------------ module functions
#define MCB_BEGIN(count)                                  \
  HANDLE_TH_ERRORS                                        \
  try {                                                   \
    check_count(n, count, __func__);

#define MCB_END                                           \
  } catch (const Failed&) {                               \
    return nullptr;                                       \
  }                                                       \
  END_HANDLE_TH_ERRORS

PyObject* mm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(10)
  const Tensor c = gemm(static_cast<int>(integer(a[0])), tensor(a[1]), tensor(a[2]), optional(a[3]), optional(a[4]),
                        truth(a[5]), truth(a[6]), real(a[7]), static_cast<int>(integer(a[8])),
                        static_cast<int>(integer(a[9])));
  return THPVariable_Wrap(c);
  MCB_END
}

PyObject* rmsnorm_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {       // x, w, eps, zc -> y, x2, rstd
  MCB_BEGIN(4)
  const Tensor& x = tensor(a[0]);
  const Tensor x2 = rows_of(x, x.size(-1));
  Tensor y, rstd;
  norm_fwd(x2, tensor(a[1]), real(a[2]), truth(a[3]), y, rstd);
  return tuple({y, x2, rstd});
  MCB_END
}

PyObject* rmsnorm_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {       // dy, x2, w, rstd, eps, zc, need_dw -> dx, dw
  MCB_BEGIN(7)
  const Tensor& x2 = tensor(a[1]);
  const Tensor dy = tensor(a[0]).reshape({x2.size(0), x2.size(1)}).contiguous();
  Tensor dx, dw;
  norm_bwd(dy, x2, tensor(a[2]), tensor(a[3]), real(a[4]), truth(a[5]), false, truth(a[6]), dx, dw);
  return tuple({dx, dw});
  MCB_END
}

PyObject* norm_linear_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {   // x, norm weight, weight, eps, zc -> y, x2, rstd
  MCB_BEGIN(5)
  const Tensor& x = tensor(a[0]);
  const Tensor x2 = rows_of(x, x.size(-1));
  Tensor xn, rstd;
  norm_fwd(x2, tensor(a[1]), real(a[3]), truth(a[4]), xn, rstd);
  const Tensor y = gemm(NT, xn, tensor(a[2]), Tensor(), Tensor(), false, false, 1.f, 0, 0);
  return tuple({y, x2, rstd});
  MCB_END
}

// dy, x2, norm weight, rstd, weight, eps, zc, need_dw -> dx, d norm weight, dy2, normalised input (with need_dw)
PyObject* norm_linear_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(8)
  const Tensor &x2 = tensor(a[1]), &w = tensor(a[4]);
  const Tensor dy2 = rows_of(tensor(a[0]), w.size(0));
  const bool need_dw = truth(a[7]);
  const Tensor dxn = gemm(NN, dy2, w, Tensor(), Tensor(), false, false, 1.f, 0, 0);
  Tensor dx, dlw;
  norm_bwd(dxn, x2, tensor(a[2]), tensor(a[3]), real(a[5]), truth(a[6]), need_dw, true, dx, dlw);
  return tuple({dx, dlw, dy2, need_dw ? dxn : Tensor()});
  MCB_END
}

PyObject* glu_linear_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {    // h, weight, kind, clamp, offset -> y, h2
  MCB_BEGIN(5)
  const Tensor& h = tensor(a[0]);
  const Tensor h2 = rows_of(h, h.size(-1));
  const ll rows = h2.size(0), F = h2.size(1) / 2;
  operand(h2, at::kBFloat16, 0, h2, "gated activation: bf16");
  const Tensor act = at::empty({rows, F}, h2.options());
  launch("mcb_glu_fwd", mcb_glu_fwd, h2.data_ptr(), nullptr, act.data_ptr(), rows, F, h2.stride(0), integer(a[2]),
         real(a[3]), real(a[4]), stream());
  return tuple({gemm(NT, act, tensor(a[1]), Tensor(), Tensor(), false, false, 1.f, 0, 0), h2});
  MCB_END
}

// dy, h2, weight, kind, clamp, offset, need_dw -> dh, dy2, activation (with need_dw)
PyObject* glu_linear_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(7)
  const Tensor &h2 = tensor(a[1]), &w = tensor(a[2]);
  const Tensor dy2 = rows_of(tensor(a[0]), w.size(0));
  const bool need_dw = truth(a[6]);
  const ll rows = h2.size(0), F2 = h2.size(1);
  const Tensor da = gemm(NN, dy2, w, Tensor(), Tensor(), false, false, 1.f, 0, 0);
  const Tensor dh = at::empty({rows, F2}, h2.options());
  const int kind = static_cast<int>(integer(a[3])), F = static_cast<int>(F2 / 2);
  const float clamp = real(a[4]), offset = real(a[5]);
  if (need_dw)
    launch("mcb_glu_bwd", mcb_glu_bwd_act, h2.data_ptr(), nullptr, da.data_ptr(), dh.data_ptr(), nullptr, rows, F, h2.stride(0),
           kind, clamp, offset, stream());
  else
    launch("mcb_glu_bwd", mcb_glu_bwd, h2.data_ptr(), nullptr, da.data_ptr(), dh.data_ptr(), nullptr, rows, F, h2.stride(0),
           kind, clamp, offset, stream());
  return tuple({dh, dy2, need_dw ? da : Tensor()});
  MCB_END
}

PyObject* glu_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {           // x, probs, kind, clamp, offset -> y, x2
  MCB_BEGIN(5)
  const Tensor& x = tensor(a[0]);
  const Tensor x2 = rows_of(x, x.size(-1)), probs = optional(a[1]);
  const ll rows = x2.size(0), F = x2.size(1) / 2;
  operand(x2, at::kBFloat16, 0, x2, "gated activation: bf16");
  operand(probs, at::kFloat, rows, x2, "gated activation: an fp32 factor for every row");
  const Tensor y = at::empty({rows, F}, x2.options());
  launch("mcb_glu_fwd", mcb_glu_fwd, x2.data_ptr(), ptr(probs), y.data_ptr(), rows, F, x2.stride(0), integer(a[2]), real(a[3]),
         real(a[4]), stream());
  return tuple({y, x2});
  MCB_END
}

PyObject* glu_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {           // dy, x2, probs, kind, clamp, offset -> dx, dprobs
  MCB_BEGIN(6)
  const Tensor& x2 = tensor(a[1]);
  const Tensor probs = optional(a[2]);
  const ll rows = x2.size(0), F2 = x2.size(1);
  const Tensor dy = tensor(a[0]).reshape({rows, F2 / 2}).contiguous();
  operand(dy, at::kBFloat16, 0, x2, "gated activation: bf16");
  operand(probs, at::kFloat, rows, x2, "gated activation: an fp32 factor for every row");
  const Tensor dx = at::empty({rows, F2}, x2.options());
  const Tensor dp = probs.defined() ? at::empty({rows}, x2.options().dtype(at::kFloat)) : Tensor();
  launch("mcb_glu_bwd", mcb_glu_bwd, x2.data_ptr(), ptr(probs), dy.data_ptr(), dx.data_ptr(), ptr(dp), rows, F2 / 2,
         x2.stride(0), integer(a[3]), real(a[4]), real(a[5]), stream());
  return tuple({dx, dp});
  MCB_END
}

void check_qkv(const Tensor& qkv, const Tensor& wq, const Tensor& wk, const Tensor& cos, const Tensor& sin, ll ng, ll qpg, ll d,
               bool gated) {
  const ll T = qkv.size(0);
  operand(qkv, at::kBFloat16, T * ng * (qpg * (gated ? 2 : 1) + 2) * d, qkv, "qkv: bf16, every head of every group");
  require(wq.defined() == wk.defined() && cos.defined() == sin.defined(), "qkv: both weights and both tables, or neither");
  operand(wq, at::kBFloat16, d, qkv, "query norm weight: bf16, one for every channel");
  operand(wk, at::kBFloat16, d, qkv, "key norm weight: bf16, one for every channel");
  operand(cos, at::kFloat, T * (cos.defined() ? cos.size(-1) : 0), qkv, "cosines: fp32, a row for every token");
  operand(sin, at::kFloat, T * (cos.defined() ? cos.size(-1) : 0), qkv, "sines: fp32, a row for every token");
}

// qkv, wq, wk, cos, sin, ng, qpg, d, has_gate, interleaved, eps, zc -> q, k, v, gate, qkv
PyObject* qkv_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(12)
  const Tensor& qkv_ = tensor(a[0]);
  const Tensor qkv = qkv_.stride(-1) == 1 ? qkv_ : qkv_.contiguous();
  const Tensor wq = optional(a[1]), wk = optional(a[2]), cos = optional(a[3]), sin = optional(a[4]);
  const ll T = qkv.size(0), ng = integer(a[5]), qpg = integer(a[6]), d = integer(a[7]);
  const bool gated = truth(a[8]);
  check_qkv(qkv, wq, wk, cos, sin, ng, qpg, d, gated);
  const Tensor q = at::empty({T, ng * qpg, d}, qkv.options()), k = at::empty({T, ng, d}, qkv.options()),
               v = at::empty({T, ng, d}, qkv.options());
  const Tensor gate = gated ? at::empty({T, ng * qpg, d}, qkv.options()) : Tensor();
  launch("mcb_qkv_split_norm_rope_fwd", mcb_qkv_split_norm_rope_fwd, qkv.data_ptr(), ptr(wq), ptr(wk), ptr(cos), ptr(sin),
         q.data_ptr(), k.data_ptr(), v.data_ptr(), ptr(gate), T, ng, qpg, d, gated, cos.defined() ? cos.size(-1) * 2 : 0,
         truth(a[9]), wq.defined(), truth(a[11]), real(a[10]), qkv.stride(0), stream());
  return tuple({q, k, v, gate, qkv});
  MCB_END
}

// dq, dk, dv, dgate, qkv, wq, wk, cos, sin, ng, qpg, d, has_gate, interleaved, eps, zc -> dqkv, dwq, dwk
PyObject* qkv_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(16)
  const Tensor& qkv = tensor(a[4]);
  const Tensor wq = optional(a[5]), wk = optional(a[6]), cos = optional(a[7]), sin = optional(a[8]);
  const ll T = qkv.size(0), ng = integer(a[9]), qpg = integer(a[10]), d = integer(a[11]);
  const bool gated = truth(a[12]), norm = wq.defined();
  check_qkv(qkv, wq, wk, cos, sin, ng, qpg, d, gated);
  auto grad = [&](PyObject* o, ll heads) {
    return o == Py_None ? at::zeros({T, heads, d}, qkv.options()) : tensor(o).contiguous();
  };
  const Tensor dq = grad(a[0], ng * qpg), dk = grad(a[1], ng), dv = grad(a[2], ng);
  const Tensor dgate = gated ? grad(a[3], ng * qpg) : Tensor();
  const Tensor dqkv = at::empty_like(qkv);
  Tensor dw, dwq, dwk, part;
  if (norm) {
    // bf16 weights (the only ones this path takes): the reduction writes them rounded; per-CTA partial sums are added in a
    // fixed order
    dw = T ? at::empty({2, d}, wq.options()) : at::zeros({2, d}, wq.options());
    dwq = dw.select(0, 0);
    dwk = dw.select(0, 1);
    part = at::empty({mcb_qkv_bwd_partial_rows(T), 2, d}, qkv.options().dtype(at::kFloat));
  }
  launch("mcb_qkv_split_norm_rope_bwd", mcb_qkv_split_norm_rope_bwd, qkv.data_ptr(), ptr(wq), ptr(wk), ptr(cos), ptr(sin),
         dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), ptr(dgate), dqkv.data_ptr(), ptr(dwq), ptr(dwk), 1, ptr(part), T, ng,
         qpg, d, gated, cos.defined() ? cos.size(-1) * 2 : 0, truth(a[13]), norm, truth(a[15]), real(a[14]), qkv.stride(0),
         stream());
  return tuple({dqkv, dwq, dwk});
  MCB_END
}

// q, k, v, k_lo, k_hi, sinks, scale -> o, lse, q, k, v (contiguous)
PyObject* attn_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(7)
  const Tensor q = tensor(a[0]).contiguous(), k = tensor(a[1]).contiguous(), v = tensor(a[2]).contiguous();
  const ll T = q.size(0), nq = q.size(1), d = q.size(2);
  operand(q, at::kBFloat16, 0, q, "queries: bf16");
  operand(k, at::kBFloat16, k.size(0) * k.size(1) * d, q, "keys: bf16 with the queries' channels");
  operand(v, at::kBFloat16, k.numel(), q, "values: bf16, as many as keys");
  const Tensor k_lo = per_token(tensor(a[3]), T, q, "first keys: an int32 for every query, on the queries' device"),
               k_hi = per_token(optional(a[4]), T, q, "last keys: an int32 for every query, on the queries' device"),
               sinks = optional(a[5]);
  operand(sinks, at::kFloat, nq, q, "sinks: an fp32 for every head");
  const Tensor o = at::empty_like(q), lse = at::empty({nq, T}, q.options().dtype(at::kFloat));
  launch("mcb_attn_fwd_ranges", mcb_attn_fwd_ranges, q.data_ptr(), k.data_ptr(), v.data_ptr(), k_lo.data_ptr(), ptr(k_hi),
         ptr(sinks), o.data_ptr(), lse.data_ptr(), T, k.size(0), nq, k.size(1), d, real(a[6]), status_of(q), stream());
  return tuple({o, lse, q, k, v});
  MCB_END
}

// do, q, k, v, o, lse, k_lo, k_hi, q_lo, q_hi, sinks, bf16 sinks, scale -> dq, dk, dv, dsinks
PyObject* attn_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(13)
  const Tensor dout = tensor(a[0]).contiguous();
  const Tensor &q = tensor(a[1]), &k = tensor(a[2]), &v = tensor(a[3]), &o = tensor(a[4]), &lse = tensor(a[5]);
  const ll T = q.size(0), Tk = k.size(0), d = q.size(2);
  const Tensor k_lo = per_token(tensor(a[6]), T, q, "first keys: an int32 for every query, on the queries' device"),
               k_hi = per_token(optional(a[7]), T, q, "last keys: an int32 for every query, on the queries' device"),
               q_lo = per_token(optional(a[8]), Tk, q, "first queries: an int32 for every key, on the keys' device"),
               q_hi = per_token(optional(a[9]), Tk, q, "last queries: an int32 for every key, on the keys' device");
  const int nq = static_cast<int>(q.size(1)), nkv = static_cast<int>(k.size(1));
  const Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  const Tensor delta = at::empty({nq, T}, lse.options());
  const int splits = dkv_splits(Tk, nq, nkv);
  const Tensor partial = splits > 1 ? at::empty({2, splits, Tk, nkv, d}, lse.options()) : Tensor();
  launch("mcb_attn_bwd_ranges", mcb_attn_bwd_ranges, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
         dout.data_ptr(), lse.data_ptr(), delta.data_ptr(), 0, k_lo.data_ptr(), ptr(k_hi), ptr(q_lo), ptr(q_hi),
         dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), T, Tk, nq, nkv, d, real(a[12]), ptr(partial), splits, status_of(q),
         stream());
  Tensor dsinks;
  if (a[10] != Py_None) {
    const Tensor& sinks = tensor(a[10]);
    const bool narrow = truth(a[11]);
    dsinks = at::empty({nq}, lse.options().dtype(narrow ? at::kBFloat16 : at::kFloat));
    launch("mcb_attn_sink_grad", mcb_attn_sink_grad, sinks.data_ptr(), lse.data_ptr(), delta.data_ptr(), dsinks.data_ptr(),
           narrow, T, nq, stream());
  }
  return tuple({dq, dk, dv, dsinks});
  MCB_END
}

PyObject* attn_window_starts(PyObject*, PyObject* const* a, Py_ssize_t n) {   // seq_start, left -> first visible keys
  MCB_BEGIN(2)
  const Tensor start = per_token(tensor(a[0]), 0, tensor(a[0]), "sequence starts: int32");
  const ll left = integer(a[1]);
  const Tensor out = at::empty_like(start);
  launch("mcb_attn_window_starts", mcb_attn_window_starts, start.data_ptr(), out.data_ptr(), start.numel(),
         left < INT32_MAX ? left : INT32_MAX, stream());
  return THPVariable_Wrap(out);
  MCB_END
}

PyObject* attn_dkv_splits(PyObject*, PyObject* const* a, Py_ssize_t n) {      // keys, query heads, kv heads
  MCB_BEGIN(3)
  return PyLong_FromLong(dkv_splits(integer(a[0]), static_cast<int>(integer(a[1])), static_cast<int>(integer(a[2]))));
  MCB_END
}

PyObject* enabled(PyObject*, PyObject*) {
  const char* e = std::getenv("MCB200_DISABLE_CUDA_KERNELS");
  return PyBool_FromLong(!(e && std::strcmp(e, "1") == 0));
}

PyObject* launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches); }

PyObject* raw_stream(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  return PyLong_FromVoidPtr(stream());
  END_HANDLE_TH_ERRORS
}

PyObject* memory(PyObject*, PyObject* const* a, Py_ssize_t n) {   // device -> bytes the caching allocator holds, and has given out
  MCB_BEGIN(1)
  const auto s = c10::cuda::CUDACachingAllocator::getDeviceStats(static_cast<c10::DeviceIndex>(integer(a[0])));
  const size_t all = static_cast<size_t>(c10::CachingAllocator::StatType::AGGREGATE);
  return Py_BuildValue("LL", static_cast<ll>(s.reserved_bytes[all].current), static_cast<ll>(s.allocated_bytes[all].current));
  MCB_END
}

PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t n) {   // path of libmcb200.so, exception class, status callback
  MCB_BEGIN(3)
  const char* path = PyUnicode_AsUTF8(a[0]);
  if (path == nullptr) return nullptr;
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (lib == nullptr) {
    PyErr_Format(PyExc_OSError, "%s", dlerror());
    return nullptr;
  }
#define MCB_RESOLVE(name, ret, args)                                       \
  name = reinterpret_cast<ret(*) args>(dlsym(lib, #name));                 \
  if (name == nullptr) {                                                   \
    PyErr_Format(PyExc_OSError, "%s has no entry point " #name, path);     \
    return nullptr;                                                        \
  }
  MCB_ENTRIES(MCB_RESOLVE)
  g_kernel_error = Py_NewRef(a[1]);
  g_make_status = Py_NewRef(a[2]);
  Py_RETURN_NONE;
  MCB_END
}

#define MCB_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {MCB_FAST(init),
                         {"enabled", enabled, METH_NOARGS, nullptr},
                         {"launches", launches, METH_NOARGS, nullptr},
                         {"raw_stream", raw_stream, METH_NOARGS, nullptr},
                         MCB_FAST(memory),
                         MCB_FAST(mm),
                         MCB_FAST(rmsnorm_fwd),
                         MCB_FAST(rmsnorm_bwd),
                         MCB_FAST(norm_linear_fwd),
                         MCB_FAST(norm_linear_bwd),
                         MCB_FAST(glu_linear_fwd),
                         MCB_FAST(glu_linear_bwd),
                         MCB_FAST(glu_fwd),
                         MCB_FAST(glu_bwd),
                         MCB_FAST(qkv_fwd),
                         MCB_FAST(qkv_bwd),
                         MCB_FAST(attn_fwd),
                         MCB_FAST(attn_bwd),
                         MCB_FAST(attn_window_starts),
                         MCB_FAST(attn_dkv_splits),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_mcb200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__mcb200_host() { return PyModule_Create(&module); }
