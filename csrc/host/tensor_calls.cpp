// The host side of the calls a training step makes most: allocation of the results, checks, launch.  A CPython module
// (mcore_bridge_b200/lib/_mcb200_host.*.so) that takes and returns tensors; the kernels are reached through the C entry points of
// libmcb200.so.  In Python, argument by argument through ctypes, a GEMM of a small model spent about 24 us on the host for 7 us
// on the device.
#include "tensor_ops.h"

#include <dlfcn.h>

#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>

#include <cstdlib>
#include <cstring>
#include <initializer_list>

namespace mcb_host {

#define MCB_DECLARE(name, ret, args) ret(*name) args = nullptr;
MCB_ENTRIES(MCB_DECLARE)

PyObject* g_kernel_error = nullptr;   // exception class
ll g_launches = 0;

namespace {
PyObject* g_make_status = nullptr;    // device index -> address of the device's status words
constexpr int MAX_DEVICES = 64;
int* g_status[MAX_DEVICES] = {nullptr};
}  // namespace

// ------------------------------------------------------------------------------------------------ helpers
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

Tensor rows_of(const Tensor& t, ll width) {           // [rows, width] with a contiguous last dimension
  Tensor r = t.dim() == 2 ? t : t.reshape({-1, width});
  return r.stride(-1) == 1 ? r : r.contiguous();
}

static Tensor tma_rows(const Tensor& t) {                    // ... whose rows TMA can address
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

void operand(const Tensor& t, at::ScalarType type, ll n, const Tensor& like, const char* what) {
  require(!t.defined() || (t.scalar_type() == type && t.numel() >= n && t.device() == like.device()), what);
}

Tensor per_token(const Tensor& t, ll n, const Tensor& like, const char* what) {
  operand(t, at::kInt, n, like, what);
  return t.defined() ? t.contiguous() : t;
}

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

bool gemm_residual(const Tensor& a_, const Tensor& b_, const Tensor& bias_, const Tensor& res, const Tensor& y) {
  const ll M = a_.size(0), K = a_.size(1), N = b_.size(0);
  auto starts = [](const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; };
  if (M == 0 || K == 0 || N % 8 || res.dim() != 2 || res.scalar_type() != at::kBFloat16 || res.stride(1) != 1 || res.stride(0) % 8 ||
      !starts(res) || !starts(y))
    return false;
  const Tensor a = tma_rows(a_), b = tma_rows(b_);
  operand(a, at::kBFloat16, M * K, a, "GEMM operands: bf16 on one device");
  operand(b, at::kBFloat16, N * K, a, "GEMM operands: bf16 on one device");
  require(b.size(1) == K, "GEMM operands whose contraction sizes differ");
  require(res.size(0) == M && res.size(1) == N && res.device() == a.device(), "residual of another shape");
  require(!bias_.defined() || (bias_.numel() == N && bias_.device() == a.device()), "GEMM bias: one for every column");
  Tensor bias = bias_;
  if (bias.defined()) bias = bias.to(at::kBFloat16).contiguous();
  launch("mcb_gemm_bf16_residual", mcb_gemm_bf16_residual, a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), y.data_ptr(), N,
         res.data_ptr(), res.stride(0), M, N, K, ptr(bias), status_of(a), stream());
  return true;
}

void norm_fwd(const Tensor& x2, const Tensor& w_, float eps, bool zc, const Tensor& y, Tensor& rstd) {
  const ll rows = x2.size(0), H = x2.size(1);
  const Tensor w = aligned(w_);
  operand(x2, at::kBFloat16, 0, x2, "norm input: bf16");
  operand(w, at::kBFloat16, H, x2, "norm weight: bf16, one for every column");
  rstd = at::empty({rows}, x2.options().dtype(at::kFloat));
  launch("mcb_rmsnorm_fwd", mcb_rmsnorm_fwd, x2.data_ptr(), nullptr, w.data_ptr(), y.data_ptr(), nullptr, rstd.data_ptr(),
         rows, H, x2.stride(0), eps, zc, stream());
}

void norm_bwd(const Tensor& dy_, const Tensor& x2, const Tensor& w_, const Tensor& rstd, float eps, bool zc, bool over,
              bool need_dw, const Tensor& dres_, Tensor& dx, Tensor& dw) {
  const ll rows = x2.size(0), H = x2.size(1);
  const Tensor dy = over ? dy_ : aligned(dy_), w = aligned(w_);   // what is replaced is a product's result
  // a wider row's kernel has no registers for it: 3000 x 12288 189 us, 114 without it and an addition of 221 MB
  const Tensor dres = H <= 8192 ? aligned(dres_) : Tensor();
  operand(dy, at::kBFloat16, rows * H, x2, "norm gradient: bf16 of the input's size");
  operand(w, at::kBFloat16, H, x2, "norm weight: bf16, one for every column");
  operand(rstd, at::kFloat, rows, x2, "norm: an fp32 for every row");
  operand(dres, at::kBFloat16, rows * H, x2, "gradient of the residual: bf16 of the input's size");
  dx = at::empty({rows, H}, x2.options());
  Tensor part;
  if (need_dw) {
    dw = rows ? at::empty({H}, w.options()) : at::zeros({H}, w.options());
    part = at::empty({mcb_rmsnorm_bwd_partial_rows(rows, static_cast<int>(H)), H}, x2.options().dtype(at::kFloat));
  }
  if (over)
    launch("mcb_rmsnorm_bwd_det", mcb_rmsnorm_bwd_det_y, dy.data_ptr(), x2.data_ptr(), w.data_ptr(), rstd.data_ptr(), ptr(dres),
           dx.data_ptr(), ptr(dw), need_dw, ptr(part), rows, H, x2.stride(0), eps, zc, stream());
  else
    launch("mcb_rmsnorm_bwd_det", mcb_rmsnorm_bwd_det_add, dy.data_ptr(), x2.data_ptr(), w.data_ptr(), rstd.data_ptr(), ptr(dres),
           dx.data_ptr(), ptr(dw), need_dw, ptr(part), rows, H, x2.stride(0), eps, zc, stream());
  if (dres_.defined() && !dres.defined()) dx = dx.add(dres_);
}

// How many CTAs share one (key tile, kv head) pair in the dK/dV kernel: the smallest divisor of the GQA ratio that puts about three
// CTAs on every SM, or the largest there is; a step of more than twice is taken only while SMs are idle.  dK/dV and the sum of
// the parts, us, whole / in 3, 3, 5 and 3 parts: 3000 tokens, 9 / 3 heads of 128 133 / 63, 8192 in seven sequences, 3 / 1 heads of 64
// 107 / 48, 777, 5 / 1 of 128 35 / 18; 4096, 24 / 8 of 64 171 / 194 (256 pairs).
// MCB200_ATTN_DKV_SPLITS overrides it.
static int dkv_splits(ll T, int nq, int nkv) {
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

Tensor glu_rows_fwd(const Tensor& x2, const Tensor& probs, const GluArgs& g) {
  const ll rows = x2.size(0), F = x2.size(1) / 2;
  operand(x2, at::kBFloat16, 0, x2, "gated activation: bf16");
  operand(probs, at::kFloat, rows, x2, "gated activation: an fp32 factor for every row");
  const Tensor y = at::empty({rows, F}, x2.options());
  launch("mcb_glu_fwd", mcb_glu_fwd, x2.data_ptr(), ptr(probs), y.data_ptr(), rows, F, x2.stride(0), g.kind, g.clamp, g.offset,
         stream());
  return y;
}

Tensor glu_rows_bwd(const Tensor& da, const Tensor& x2, const Tensor& probs, const GluArgs& g, bool over, Tensor& dprobs) {
  const ll rows = x2.size(0), F2 = x2.size(1);
  operand(da, at::kBFloat16, rows * (F2 / 2), x2, "gated activation: bf16");
  operand(probs, at::kFloat, rows, x2, "gated activation: an fp32 factor for every row");
  const Tensor dx = at::empty({rows, F2}, x2.options());
  if (probs.defined()) dprobs = at::empty({rows}, x2.options().dtype(at::kFloat));
  if (over)
    launch("mcb_glu_bwd", mcb_glu_bwd_act, x2.data_ptr(), ptr(probs), da.data_ptr(), dx.data_ptr(), ptr(dprobs), rows, F2 / 2,
           x2.stride(0), g.kind, g.clamp, g.offset, stream());
  else
    launch("mcb_glu_bwd", mcb_glu_bwd, x2.data_ptr(), ptr(probs), da.data_ptr(), dx.data_ptr(), ptr(dprobs), rows, F2 / 2,
           x2.stride(0), g.kind, g.clamp, g.offset, stream());
  return dx;
}

static void check_qkv(const Tensor& qkv, const Tensor& wq, const Tensor& wk, const Tensor& cos, const Tensor& sin, const QkvArgs& g) {
  const ll T = qkv.size(0), d = g.d;
  operand(qkv, at::kBFloat16, T * g.ng * (g.qpg * (g.gated ? 2 : 1) + 2) * d, qkv, "qkv: bf16, every head of every group");
  require(wq.defined() == wk.defined() && cos.defined() == sin.defined(), "qkv: both weights and both tables, or neither");
  operand(wq, at::kBFloat16, d, qkv, "query norm weight: bf16, one for every channel");
  operand(wk, at::kBFloat16, d, qkv, "key norm weight: bf16, one for every channel");
  operand(cos, at::kFloat, T * (cos.defined() ? cos.size(-1) : 0), qkv, "cosines: fp32, a row for every token");
  operand(sin, at::kFloat, T * (cos.defined() ? cos.size(-1) : 0), qkv, "sines: fp32, a row for every token");
}

Qkv qkv_split(const Tensor& qkv, const Tensor& wq_, const Tensor& wk_, const Tensor& cos_, const Tensor& sin_, const QkvArgs& g) {
  check_qkv(qkv, wq_, wk_, cos_, sin_, g);
  const Tensor wq = aligned(wq_, 4), wk = aligned(wk_, 4), cos = aligned(cos_, 8), sin = aligned(sin_, 8);
  const ll T = qkv.size(0), d = g.d;
  Qkv r;
  r.q = at::empty({T, g.ng * g.qpg, d}, qkv.options());
  r.k = at::empty({T, g.ng, d}, qkv.options());
  r.v = at::empty({T, g.ng, d}, qkv.options());
  if (g.gated) r.gate = at::empty({T, g.ng * g.qpg, d}, qkv.options());
  launch("mcb_qkv_split_norm_rope_fwd", mcb_qkv_split_norm_rope_fwd, qkv.data_ptr(), ptr(wq), ptr(wk), ptr(cos), ptr(sin),
         r.q.data_ptr(), r.k.data_ptr(), r.v.data_ptr(), ptr(r.gate), T, g.ng, g.qpg, d, g.gated,
         cos.defined() ? cos.size(-1) * 2 : 0, g.interleaved, wq.defined(), g.zc, g.eps, qkv.stride(0), stream());
  return r;
}

void qkv_join(Qkv dr, const Tensor& qkv_, const Tensor& wq_, const Tensor& wk_, const Tensor& cos_, const Tensor& sin_, const QkvArgs& g,
              Tensor& dqkv, Tensor& dwq, Tensor& dwk) {
  // the kernels write the gradient with the strides they read qkv by: columns of a wider tensor are copied first
  const Tensor qkv = qkv_.contiguous();
  const ll T = qkv.size(0), d = g.d;
  check_qkv(qkv, wq_, wk_, cos_, sin_, g);
  const Tensor wq = aligned(wq_, 4), wk = aligned(wk_, 4), cos = aligned(cos_, 8), sin = aligned(sin_, 8);
  const bool norm = wq.defined();
  const int bytes = qkv_boundary(g, cos);
  auto grad = [&](const Tensor& t, ll heads) {
    return t.defined() ? aligned(t.contiguous(), bytes) : at::zeros({T, heads, d}, qkv.options());
  };
  const Tensor dq = grad(dr.q, g.ng * g.qpg), dk = grad(dr.k, g.ng), dv = grad(dr.v, g.ng);
  const Tensor dgate = g.gated ? grad(dr.gate, g.ng * g.qpg) : Tensor();
  dqkv = at::empty_like(qkv);
  Tensor part;
  if (norm) {
    // bf16 weights (the only ones this path takes): the reduction writes them rounded; per-CTA partial sums are added in a
    // fixed order
    const Tensor dw = T ? at::empty({2, d}, wq.options()) : at::zeros({2, d}, wq.options());
    dwq = dw.select(0, 0);
    dwk = dw.select(0, 1);
    part = at::empty({mcb_qkv_bwd_partial_rows(T), 2, d}, qkv.options().dtype(at::kFloat));
  }
  launch("mcb_qkv_split_norm_rope_bwd", mcb_qkv_split_norm_rope_bwd, qkv.data_ptr(), ptr(wq), ptr(wk), ptr(cos), ptr(sin),
         dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), ptr(dgate), dqkv.data_ptr(), ptr(dwq), ptr(dwk), 1, ptr(part), T, g.ng,
         g.qpg, d, g.gated, cos.defined() ? cos.size(-1) * 2 : 0, g.interleaved, norm, g.zc, g.eps, qkv.stride(0), stream());
}

void attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k_lo_, const Tensor& k_hi_, const Tensor& sinks,
                  float scale, Tensor& o, Tensor& lse) {
  const ll T = q.size(0), nq = q.size(1), d = q.size(2);
  operand(q, at::kBFloat16, 0, q, "queries: bf16");
  operand(k, at::kBFloat16, k.size(0) * k.size(1) * d, q, "keys: bf16 with the queries' channels");
  operand(v, at::kBFloat16, k.numel(), q, "values: bf16, as many as keys");
  const Tensor k_lo = per_token(k_lo_, T, q, "first keys: an int32 for every query, on the queries' device"),
               k_hi = per_token(k_hi_, T, q, "last keys: an int32 for every query, on the queries' device");
  operand(sinks, at::kFloat, nq, q, "sinks: an fp32 for every head");
  o = at::empty_like(q);
  lse = at::empty({nq, T}, q.options().dtype(at::kFloat));
  launch("mcb_attn_fwd_ranges", mcb_attn_fwd_ranges, q.data_ptr(), k.data_ptr(), v.data_ptr(), k_lo.data_ptr(), ptr(k_hi),
         ptr(sinks), o.data_ptr(), lse.data_ptr(), T, k.size(0), nq, k.size(1), d, scale, status_of(q), stream());
}

AttnGrads attn_backward(const Tensor& dout_, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                        const Tensor& k_lo_, const Tensor& k_hi_, const Tensor& q_lo_, const Tensor& q_hi_, const Tensor& sinks,
                        bool narrow_sinks, float scale) {
  const Tensor dout = dout_.contiguous();
  const ll T = q.size(0), Tk = k.size(0), d = q.size(2);
  const Tensor k_lo = per_token(k_lo_, T, q, "first keys: an int32 for every query, on the queries' device"),
               k_hi = per_token(k_hi_, T, q, "last keys: an int32 for every query, on the queries' device"),
               q_lo = per_token(q_lo_, Tk, q, "first queries: an int32 for every key, on the keys' device"),
               q_hi = per_token(q_hi_, Tk, q, "last queries: an int32 for every key, on the keys' device");
  const int nq = static_cast<int>(q.size(1)), nkv = static_cast<int>(k.size(1));
  AttnGrads g{at::empty_like(q), at::empty_like(k), at::empty_like(v), {}};
  const Tensor delta = at::empty({nq, T}, lse.options());
  const int splits = dkv_splits(Tk, nq, nkv);
  const Tensor partial = splits > 1 ? at::empty({2, splits, Tk, nkv, d}, lse.options()) : Tensor();
  launch("mcb_attn_bwd_ranges", mcb_attn_bwd_ranges, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
         dout.data_ptr(), lse.data_ptr(), delta.data_ptr(), 0, k_lo.data_ptr(), ptr(k_hi), ptr(q_lo), ptr(q_hi),
         g.dq.data_ptr(), g.dk.data_ptr(), g.dv.data_ptr(), T, Tk, nq, nkv, d, scale, ptr(partial), splits, status_of(q), stream());
  if (sinks.defined()) {
    g.dsinks = at::empty({nq}, lse.options().dtype(narrow_sinks ? at::kBFloat16 : at::kFloat));
    launch("mcb_attn_sink_grad", mcb_attn_sink_grad, sinks.data_ptr(), lse.data_ptr(), delta.data_ptr(), g.dsinks.data_ptr(),
           narrow_sinks, T, nq, stream());
  }
  return g;
}

// ------------------------------------------------------------------------------------------------ module functions
namespace {

PyObject* mm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(10)
  const Tensor c = gemm(static_cast<int>(integer(a[0])), tensor(a[1]), tensor(a[2]), optional(a[3]), optional(a[4]),
                        truth(a[5]), truth(a[6]), real(a[7]), static_cast<int>(integer(a[8])),
                        static_cast<int>(integer(a[9])));
  return THPVariable_Wrap(c);
  MCB_END
}

GluArgs glu_args(PyObject* const* a) { return {static_cast<int>(integer(a[0])), real(a[1]), real(a[2])}; }

PyObject* glu_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {           // x, probs, kind, clamp, offset -> y, x2
  MCB_BEGIN(5)
  const Tensor& x = tensor(a[0]);
  const Tensor x2 = aligned(rows_of(x, x.size(-1)));
  return tuple({glu_rows_fwd(x2, optional(a[1]), glu_args(a + 2)), x2});
  MCB_END
}

PyObject* glu_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {           // dy, x2, probs, kind, clamp, offset -> dx, dprobs
  MCB_BEGIN(6)
  const Tensor& x2 = tensor(a[1]);
  const Tensor dy = aligned(tensor(a[0]).reshape({x2.size(0), x2.size(1) / 2}).contiguous());
  Tensor dp;
  const Tensor dx = glu_rows_bwd(dy, x2, optional(a[2]), glu_args(a + 3), false, dp);
  return tuple({dx, dp});
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

PyObject* seq_starts(PyObject*, PyObject* const* a, Py_ssize_t n) {          // boundaries, tokens -> first token of each one's sequence
  MCB_BEGIN(2)
  const Tensor cu = tensor(a[0]).contiguous();
  const ll T = integer(a[1]);
  require(cu.scalar_type() == at::kInt || cu.scalar_type() == at::kLong, "sequence boundaries: int32 or int64");
  const c10::cuda::OptionalCUDAGuard here(at::device_of(cu));   // as a tensor operation: on the tensor's device
  const Tensor out = at::empty({T}, cu.options().dtype(at::kInt));
  launch("mcb_seq_starts", mcb_seq_starts, cu.data_ptr(), cu.scalar_type() == at::kLong, cu.numel(), out.data_ptr(), T, stream());
  return THPVariable_Wrap(out);
  MCB_END
}

PyObject* rope_tables(PyObject*, PyObject* const* a, Py_ssize_t n) {         // positions, inverse frequencies, scale -> cos, sin
  MCB_BEGIN(3)
  const Tensor pos = tensor(a[0]).contiguous(), inv = tensor(a[1]).contiguous();
  require(pos.scalar_type() == at::kInt || pos.scalar_type() == at::kLong, "positions: int32 or int64");
  operand(inv, at::kFloat, 0, pos, "inverse frequencies: fp32 on the positions' device");
  const c10::cuda::OptionalCUDAGuard here(at::device_of(pos));
  const ll T = pos.numel(), R = inv.numel();
  const Tensor cos = at::empty({T, R}, inv.options()), sin = at::empty({T, R}, inv.options());
  launch("mcb_rope_tables", mcb_rope_tables, pos.data_ptr(), pos.scalar_type() == at::kLong, inv.data_ptr(), real(a[2]),
         cos.data_ptr(), sin.data_ptr(), T, R, stream());
  return tuple({cos, sin});
  MCB_END
}

PyObject* ce_combine(PyObject*, PyObject* const* a, Py_ssize_t n) {          // statistics of every row's tiles -> max, sum
  MCB_BEGIN(1)
  const Tensor& part = tensor(a[0]);
  require(part.dim() == 3 && part.size(2) == 2 && part.scalar_type() == at::kFloat && part.is_contiguous(),
          "statistics: fp32 pairs of every tile of every row");
  const Tensor m = at::empty({part.size(0)}, part.options()), s = at::empty({part.size(0)}, part.options());
  launch("mcb_ce_combine", mcb_ce_combine, part.data_ptr(), m.data_ptr(), s.data_ptr(), part.size(0), part.size(1), stream());
  return tuple({m, s});
  MCB_END
}

PyObject* ce_loss(PyObject*, PyObject* const* a, Py_ssize_t n) {             // max, sum, label logits -> log-sum-exp, loss
  MCB_BEGIN(3)
  const Tensor m = tensor(a[0]).contiguous(), s = tensor(a[1]).contiguous(), tgt = tensor(a[2]).contiguous();
  for (const Tensor& t : {m, s, tgt}) operand(t, at::kFloat, m.numel(), m, "statistics: an fp32 for every row");
  const Tensor lse = at::empty_like(m), loss = at::empty_like(m);
  launch("mcb_ce_loss", mcb_ce_loss, m.data_ptr(), s.data_ptr(), tgt.data_ptr(), lse.data_ptr(), loss.data_ptr(), m.numel(), stream());
  return tuple({lse, loss});
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
                         MCB_FAST(glu_fwd),
                         MCB_FAST(glu_bwd),
                         MCB_FAST(attn_window_starts),
                         MCB_FAST(attn_dkv_splits),
                         MCB_FAST(seq_starts),
                         MCB_FAST(rope_tables),
                         MCB_FAST(ce_combine),
                         MCB_FAST(ce_loss),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_mcb200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace mcb_host

PyMODINIT_FUNC PyInit__mcb200_host() {
  PyObject* m = PyModule_Create(&mcb_host::module);
  if (m != nullptr && PyModule_AddFunctions(m, mcb_host::autograd_methods) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
