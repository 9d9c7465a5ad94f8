// The operations of the host module: tensors in, tensors out, allocation, checks and launches; shared by the calls without a
// gradient (tensor_calls.cpp) and the differentiable ones (autograd_functions.cpp).
//
// Everything runs on the calling thread's current device and stream, with the interpreter's lock held except during a launch.
// A tensor's type, device and size are checked here against what the kernel reads; the first operand's device and the sizes a
// kernel supports are the Python callers' and the C entry points' to check.
#pragma once
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace mcb_host {

using at::Tensor;
typedef long long ll;

// ------------------------------------------------------------------------------------------------ entry points
#define MCB_ENTRIES(X)                                                                                                  \
  X(mcb_gemm_bf16, int, (const void*, ll, ll, ll, int, const void*, ll, ll, ll, int, void*, ll, ll, int, int, int, int, int,  \
                         float, const void*, int, int, const int*, int, int*, int, int, void*))                         \
  X(mcb_gemm_bf16_residual, int, (const void*, ll, const void*, ll, void*, ll, const void*, ll, int, int, int, const void*,   \
                                  int*, void*))                                                                         \
  X(mcb_rmsnorm_fwd, int, (const void*, const void*, const void*, void*, void*, float*, ll, int, ll, float, int, void*))  \
  X(mcb_rmsnorm_bwd_det_add, int, (const void*, const void*, const void*, const float*, const void*, void*, void*, int, float*,   \
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
  X(mcb_seq_starts, int, (const void*, int, int, int*, ll, void*))                                                      \
  X(mcb_rope_tables, int, (const void*, int, const float*, float, float*, float*, ll, int, void*))                      \
  X(mcb_ce_combine, int, (const float*, float*, float*, ll, int, void*))                                                \
  X(mcb_ce_loss, int, (const float*, const float*, const float*, float*, float*, ll, void*))                            \
  X(mcb_sm_count, int, ())

#define MCB_EXTERN(name, ret, args) extern ret(*name) args;
MCB_ENTRIES(MCB_EXTERN)

// ------------------------------------------------------------------------------------------------ arguments and launches
struct Failed {};   // a Python exception is set

extern ll g_launches;
extern PyObject* g_kernel_error;

void check_count(Py_ssize_t got, Py_ssize_t want, const char* what);
const Tensor& tensor(PyObject* o);
Tensor optional(PyObject* o);   // None: undefined
ll integer(PyObject* o);
float real(PyObject* o);
bool truth(PyObject* o);
void require(bool ok, const char* what);
int* status_of(const Tensor& t);
inline void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
Tensor rows_of(const Tensor& t, ll width);   // [rows, width] with a contiguous last dimension
// What a kernel reads `bytes` at a time: a tensor that does not start on such a boundary is copied.
inline Tensor aligned(const Tensor& t, int bytes = 16) {
  return t.defined() && reinterpret_cast<uintptr_t>(t.data_ptr()) % bytes ? t.clone(at::MemoryFormat::Contiguous) : t;
}
// An operand a kernel reads at least n elements of one type from, beside `like`; an undefined one is left out.
void operand(const Tensor& t, at::ScalarType type, ll n, const Tensor& like, const char* what);
// What a kernel reads one int32 of per query or key from.
Tensor per_token(const Tensor& t, ll n, const Tensor& like, const char* what);
PyObject* tuple(std::initializer_list<Tensor> ts);

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

#define MCB_BEGIN(count)                                  \
  HANDLE_TH_ERRORS                                        \
  try {                                                   \
    ::mcb_host::check_count(n, count, __func__);

#define MCB_END                                           \
  } catch (const ::mcb_host::Failed&) {                   \
    return nullptr;                                       \
  }                                                       \
  END_HANDLE_TH_ERRORS

// ------------------------------------------------------------------------------------------------ operations
enum Layout { NT = 0, NN = 1, TN = 2 };

// c = op(a) . op(b): NT a [M, K], b [N, K]; NN a [M, K], b [K, N]; TN a [K, M], b [K, N]
Tensor gemm(int layout, const Tensor& a, const Tensor& b, const Tensor& bias = {}, const Tensor& out = {}, bool fp32 = false,
            bool accumulate = false, float alpha = 1.f, int max_sms = 0, int force_bn = 0);
void norm_fwd(const Tensor& x2, const Tensor& w, float eps, bool zc, const Tensor& y, Tensor& rstd);
// `over` replaces dy with the norm's result; `dres` (optional, [rows, H]) is added to the rounded dx
void norm_bwd(const Tensor& dy, const Tensor& x2, const Tensor& w, const Tensor& rstd, float eps, bool zc, bool over, bool need_dw,
              const Tensor& dres, Tensor& dx, Tensor& dw);
// y = res + a . b^T (+ bias) in the kernel's epilogue; false where the kernel does not take the operands
bool gemm_residual(const Tensor& a, const Tensor& b, const Tensor& bias, const Tensor& res, const Tensor& y);
struct GluArgs {
  int kind;
  float clamp, offset;
};
Tensor glu_rows_fwd(const Tensor& x2, const Tensor& probs, const GluArgs& g);
// with `over` da becomes the activation
Tensor glu_rows_bwd(const Tensor& da, const Tensor& x2, const Tensor& probs, const GluArgs& g, bool over, Tensor& dprobs);
struct QkvArgs {
  ll ng, qpg, d;
  bool gated, interleaved;
  float eps;
  bool zc;
};
struct Qkv {
  Tensor q, k, v, gate;
};
// The boundary its kernels want qkv and the gradients on: heads of 128 have one that reads 4 bytes where it has to.
inline int qkv_boundary(const QkvArgs& g, const Tensor& cos) {
  const ll pairs = (g.ng * (g.qpg * (g.gated ? 2 : 1) + 2) + 1) / 2;
  return g.d == 128 && cos.defined() && cos.size(-1) == 64 && !g.interleaved && pairs <= 24ll * mcb_sm_count() ? 4 : 16;
}
Qkv qkv_split(const Tensor& qkv, const Tensor& wq, const Tensor& wk, const Tensor& cos, const Tensor& sin, const QkvArgs& g);
// undefined gradients count as zero
void qkv_join(Qkv d, const Tensor& qkv, const Tensor& wq, const Tensor& wk, const Tensor& cos, const Tensor& sin, const QkvArgs& g,
              Tensor& dqkv, Tensor& dwq, Tensor& dwk);
// contiguous q, k, v
void attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& k_lo, const Tensor& k_hi, const Tensor& sinks,
                  float scale, Tensor& o, Tensor& lse);
struct AttnGrads {
  Tensor dq, dk, dv, dsinks;
};
AttnGrads attn_backward(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                        const Tensor& k_lo, const Tensor& k_hi, const Tensor& q_lo, const Tensor& q_hi, const Tensor& sinks,
                        bool narrow_sinks, float scale);

extern PyMethodDef autograd_methods[];   // ends with a null entry

}  // namespace mcb_host
