// The differentiable operations of a layer as autograd nodes of their own: a forward call builds its node here, and the backward pass
// runs it without a Python frame.  As torch.autograd.Function in Python each operation spent about 15 us a direction around the
// kernels' own launches: the forward pass of a 4-layer model of 256 channels and 201 tokens 939 -> 673 us, a training pass of 1024
// tokens 2618 -> 2096.
//
// A node keeps what the Python functions kept, by SavedVariable: hooks on saved tensors, in-place checks and "a second time" errors
// are torch's.  The nodes have no forward-mode and no vmap form and refuse both, and their results are not differentiable
// again, as before.  A weight's gradient goes to its `main_grad` where it has one, see weight_grad.
#include "tensor_ops.h"

#include <ATen/FuncTorchTLS.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <vector>

namespace mcb_host {
namespace {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------------ nodes
struct Gil {
  PyGILState_STATE s = PyGILState_Ensure();
  ~Gil() { PyGILState_Release(s); }
};

// A backward function whose body may leave a Python exception.
struct OpNode : Node {
  std::vector<SavedVariable> saved;

  virtual variable_list grads(variable_list& g) = 0;

  variable_list apply(variable_list&& g) override {
    bool any = false;
    for (const Tensor& t : g) any |= t.defined();
    if (!any) return variable_list(num_outputs());
    Gil gil;
    try {
      return grads(g);
    } catch (const Failed&) {
      python_error e;
      e.persist();
      throw e;
    }
  }
  Tensor get(size_t i) { return saved[i].unpack(shared_from_this()); }
  void save(std::initializer_list<Tensor> ts) {
    saved.reserve(ts.size() + 1);
    for (const Tensor& t : ts) saved.emplace_back(t, false);
  }
  void release_variables() override {
    for (SavedVariable& s : saved) s.reset_data();
  }
};

// What the inputs allow: plain tensors; with a gradient wanted the result needs a node.
bool wants_gradient(std::initializer_list<Tensor> inputs) {
  auto& functorch = at::functorch::functorchTLSAccessor();
  if (functorch) functorch->checkSupportsCppAutogradFunction();
  bool any = false;
  for (const Tensor& t : inputs) {
    if (!t.defined()) continue;
    TORCH_CHECK_NOT_IMPLEMENTED(!t._fw_grad(0).defined(), "forward-mode differentiation of the kernels' operations");
    any |= t.requires_grad();
  }
  return any && at::GradMode::is_enabled();
}

template <class N>
std::shared_ptr<N> make_node(std::initializer_list<Tensor> inputs) {
  std::shared_ptr<N> node(new N(), torch::autograd::deleteNode);
  torch::autograd::edge_list edges;
  edges.reserve(inputs.size());
  for (const Tensor& t : inputs) edges.push_back(t.defined() ? torch::autograd::impl::gradient_edge(t) : torch::autograd::Edge());
  node->set_next_edges(std::move(edges));
  return node;
}

// An attribute of a tensor's Python object; null where it is missing or None.
PyObject* attribute(PyObject* o, const char* name) {
  PyObject* v = PyObject_GetAttrString(o, name);
  if (v == nullptr) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw Failed();
    PyErr_Clear();
  } else if (v == Py_None) {
    Py_DECREF(v);
    v = nullptr;
  }
  return v;
}
struct Ref {
  PyObject* o;
  ~Ref() { Py_XDECREF(o); }
};

// dW = dy^T x: into the weight's `main_grad` (fp32, summed by the GEMM's epilogue; `grad_ready_hook` is told), where the optimizer
// has given it one, else returned.
Tensor weight_grad(const Tensor& weight, const Tensor& dy2, const Tensor& x2) {
  Ref w{THPVariable_Wrap(weight)};
  if (w.o == nullptr) throw Failed();
  Ref main{attribute(w.o, "main_grad")};
  if (main.o == nullptr) return gemm(TN, dy2, x2, {}, {}, weight.scalar_type() == at::kFloat);
  gemm(TN, dy2, x2, {}, tensor(main.o), false, true);
  Ref hook{attribute(w.o, "grad_ready_hook")};
  if (hook.o != nullptr) {
    Ref r{PyObject_CallNoArgs(hook.o)};
    if (r.o == nullptr) throw Failed();
  }
  return {};
}

std::vector<int64_t> with_last(const Tensor& x, ll n) {
  std::vector<int64_t> shape = x.sizes().vec();
  shape.back() = n;
  return shape;
}
Tensor like_input(const Tensor& dx, const std::vector<int64_t>& shape) { return dx.dim() == 2 && shape.size() == 2 ? dx : dx.view(shape); }
// x2 . weight^T (+ bias) (+ residual) in x's leading shape; a residual has that shape too.  One of another type is added as torch
// adds it, in the wider of the two.
Tensor product(const Tensor& x2, const Tensor& weight, const Tensor& bias, const Tensor& x, const Tensor& residual = {}) {
  const Tensor y = at::empty(with_last(x, weight.size(0)), x.options());
  if (!residual.defined()) {
    gemm(NT, x2, weight, bias, y);
    return y;
  }
  require(residual.sizes() == y.sizes(), "residual of another shape");
  const Tensor r2 = residual.dim() == 2 ? residual : residual.reshape({-1, residual.size(-1)});
  if (gemm_residual(x2, weight, bias, r2, y)) return y;
  gemm(NT, x2, weight, bias, y);
  return residual.add(y);
}

// ------------------------------------------------------------------------------------------------ linear
struct LinearNode : OpNode {
  bool need_dx, need_dw, bias, residual;
  std::vector<int64_t> shape;
  std::string name() const override { return "McbLinearBackward"; }
  variable_list grads(variable_list& g) override {
    const Tensor x2 = get(0), w = get(1);
    const Tensor dy2 = rows_of(g[0].to(w.scalar_type()), w.size(0));   // a residual may have made the result wider
    variable_list r(4);
    if (residual) r[3] = g[0];
    if (need_dx) r[0] = gemm(NN, dy2, w).view(shape);
    if (need_dw) r[1] = weight_grad(w, dy2, x2);
    if (bias) r[2] = dy2.to(at::kFloat).sum(0).to(dy2.scalar_type());
    return r;
  }
};

// x, weight, bias, skip the weight's gradient, residual -> y
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(5)
  const Tensor &x = tensor(a[0]), &w = tensor(a[1]);
  const Tensor bias = optional(a[2]), residual = optional(a[4]);
  const bool grad = wants_gradient({x, w, bias, residual});
  Tensor y, x2;
  {
    at::NoGradGuard none;
    x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
    y = product(x2, w, bias, x, residual);
  }
  if (grad) {
    auto node = make_node<LinearNode>({x, w, bias, residual});
    node->need_dx = x.requires_grad();
    node->need_dw = w.requires_grad() && !truth(a[3]);
    node->bias = bias.defined();
    node->residual = residual.defined();
    node->shape = x.sizes().vec();
    node->save({x2, w});
    torch::autograd::set_history(y, node);
  }
  return THPVariable_Wrap(y);
  MCB_END
}

// ------------------------------------------------------------------------------------------------ norm, norm + linear
struct NormNode : OpNode {
  float eps;
  bool zc, need_dw;
  std::vector<int64_t> shape;
  std::string name() const override { return "McbRMSNormBackward"; }
  variable_list grads(variable_list& g) override {
    const Tensor x2 = get(0), w = get(1), rstd = get(2);
    Tensor dx, dw;
    norm_bwd(g[0].reshape({x2.size(0), x2.size(1)}).contiguous(), x2, w, rstd, eps, zc, false, need_dw, {}, dx, dw);
    return {like_input(dx, shape), dw};
  }
};

PyObject* rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {   // x, weight, eps, zc -> y
  MCB_BEGIN(4)
  const Tensor &x = tensor(a[0]), &w = tensor(a[1]);
  const float eps = real(a[2]);
  const bool zc = truth(a[3]), grad = wants_gradient({x, w});
  Tensor y, x2, rstd;
  {
    at::NoGradGuard none;
    x2 = aligned(rows_of(x, x.size(-1)));
    y = at::empty(x.sizes(), x.options());
    norm_fwd(x2, w, eps, zc, y, rstd);
  }
  if (grad) {
    auto node = make_node<NormNode>({x, w});
    node->eps = eps;
    node->zc = zc;
    node->need_dw = w.requires_grad();
    node->shape = x.sizes().vec();
    node->save({x2, w, rstd});
    torch::autograd::set_history(y, node);
  }
  return THPVariable_Wrap(y);
  MCB_END
}

struct NormLinearNode : OpNode {
  float eps;
  bool zc, need_dw;
  std::vector<int64_t> shape;
  std::string name() const override { return "McbNormLinearBackward"; }
  variable_list grads(variable_list& g) override {
    const Tensor x2 = get(0), ln_w = get(1), rstd = get(2), w = get(3);
    if (!g[0].defined()) return {g[1], {}, {}};
    const Tensor dy2 = rows_of(g[0], w.size(0)), dxn = gemm(NN, dy2, w);
    const Tensor dkept = g.size() > 1 && g[1].defined() ? g[1].reshape({x2.size(0), x2.size(1)}).contiguous() : Tensor();
    Tensor dx, dlw;
    norm_bwd(dxn, x2, ln_w, rstd, eps, zc, need_dw, true, dkept, dx, dlw);   // dxn becomes the normalised input
    return {like_input(dx, shape), dlw, need_dw ? weight_grad(w, dy2, dxn) : Tensor()};
  }
};

// x, norm weight, weight, eps, zc, keep -> y, or with `keep` y and x again: what uses x from there sends its gradient through this
// node, whose kernel adds it to the norm's
PyObject* norm_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(6)
  const Tensor &x = tensor(a[0]), &ln_w = tensor(a[1]), &w = tensor(a[2]);
  const float eps = real(a[3]);
  const bool zc = truth(a[4]), grad = wants_gradient({x, ln_w, w});
  Tensor y, x2, rstd;
  {
    at::NoGradGuard none;
    x2 = aligned(rows_of(x, x.size(-1)));
    const Tensor xn = at::empty_like(x2, at::MemoryFormat::Contiguous);
    norm_fwd(x2, ln_w, eps, zc, xn, rstd);
    y = product(xn, w, {}, x);
  }
  if (grad) {
    auto node = make_node<NormLinearNode>({x, ln_w, w});
    node->eps = eps;
    node->zc = zc;
    node->need_dw = w.requires_grad();
    node->shape = x.sizes().vec();
    node->save({x2, ln_w, rstd, w});
    torch::autograd::set_history(y, node);
    if (truth(a[5])) {
      Tensor kept;
      {
        at::AutoDispatchBelowADInplaceOrView plain;
        kept = x.detach();
      }
      torch::autograd::set_history(kept, node);
      return tuple({y, kept});
    }
  }
  return truth(a[5]) ? tuple({y, x}) : THPVariable_Wrap(y);
  MCB_END
}

// ------------------------------------------------------------------------------------------------ gated activation + linear
struct GluLinearNode : OpNode {
  GluArgs args;
  bool need_dw, residual;
  std::vector<int64_t> shape;
  std::string name() const override { return "McbGluLinearBackward"; }
  variable_list grads(variable_list& g) override {
    const Tensor h2 = get(0), w = get(1);
    const Tensor dy2 = rows_of(g[0].to(w.scalar_type()), w.size(0)), da = gemm(NN, dy2, w);
    Tensor none;
    const Tensor dh = glu_rows_bwd(da, h2, {}, args, need_dw, none);  // da becomes the activation
    return {like_input(dh, shape), need_dw ? weight_grad(w, dy2, da) : Tensor(), residual ? g[0] : Tensor()};
  }
};

PyObject* glu_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {   // h, weight, kind, clamp, offset, residual -> y
  MCB_BEGIN(6)
  const Tensor &h = tensor(a[0]), &w = tensor(a[1]);
  const Tensor residual = optional(a[5]);
  const GluArgs args{static_cast<int>(integer(a[2])), real(a[3]), real(a[4])};
  const bool grad = wants_gradient({h, w, residual});
  Tensor y, h2;
  {
    at::NoGradGuard none;
    h2 = aligned(rows_of(h, h.size(-1)));
    y = product(glu_rows_fwd(h2, {}, args), w, {}, h, residual);
  }
  if (grad) {
    auto node = make_node<GluLinearNode>({h, w, residual});
    node->args = args;
    node->need_dw = w.requires_grad();
    node->residual = residual.defined();
    node->shape = h.sizes().vec();
    node->save({h2, w});
    torch::autograd::set_history(y, node);
  }
  return THPVariable_Wrap(y);
  MCB_END
}

// ------------------------------------------------------------------------------------------------ qkv
struct QkvNode : OpNode {
  QkvArgs args;
  std::string name() const override { return "McbQkvBackward"; }
  variable_list grads(variable_list& g) override {
    const Tensor qkv = get(0), wq = get(1), wk = get(2), cos = get(3), sin = get(4);
    Tensor dqkv, dwq, dwk;
    qkv_join({g[0], g[1], g[2], g.size() > 3 ? g[3] : Tensor()}, qkv, wq, wk, cos, sin, args, dqkv, dwq, dwk);
    return {dqkv, dwq, dwk};
  }
};

// qkv, wq, wk, cos, sin, ng, qpg, d, has_gate, interleaved, eps, zc -> q, k, v, gate
PyObject* qkv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(12)
  const Tensor& x = tensor(a[0]);
  const Tensor wq = optional(a[1]), wk = optional(a[2]), cos = optional(a[3]), sin = optional(a[4]);
  const QkvArgs args{integer(a[5]), integer(a[6]), integer(a[7]), truth(a[8]), truth(a[9]), real(a[10]), truth(a[11])};
  const bool grad = wants_gradient({x, wq, wk});
  Qkv r;
  Tensor x2;
  {
    at::NoGradGuard none;
    x2 = aligned(x.stride(-1) == 1 ? x : x.contiguous(), qkv_boundary(args, cos));
    r = qkv_split(x2, wq, wk, cos, sin, args);
  }
  if (grad) {
    auto node = make_node<QkvNode>({x, wq, wk});
    node->args = args;
    node->save({x2, wq, wk, cos, sin});
    for (Tensor* t : {&r.q, &r.k, &r.v, &r.gate})
      if (t->defined()) torch::autograd::set_history(*t, node);
  }
  return tuple({r.q, r.k, r.v, r.gate});
  MCB_END
}

// ------------------------------------------------------------------------------------------------ attention
struct AttnNode : OpNode {
  float scale;
  bool narrow_sinks = false;
  at::ScalarType sink_type = at::kFloat;
  std::string name() const override { return "McbAttentionBackward"; }
  variable_list grads(variable_list& g) override {
    const Tensor q = get(0), k = get(1), v = get(2), lse = get(3), k_lo = get(4), k_hi = get(5), q_lo = get(6), q_hi = get(7),
                 sinks = get(8), o = get(9);
    AttnGrads d = attn_backward(g[0].defined() ? g[0] : at::zeros_like(o), q, k, v, o, lse, k_lo, k_hi, q_lo, q_hi, sinks, narrow_sinks,
                                scale);
    return {d.dq, d.dk, d.dv, d.dsinks.defined() ? d.dsinks.to(sink_type) : Tensor()};
  }
};

// q, k, v, k_lo, k_hi, q_lo, q_hi, sinks, scale -> o, lse (which carries no gradient)
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  MCB_BEGIN(9)
  const Tensor &q_ = tensor(a[0]), &k_ = tensor(a[1]), &v_ = tensor(a[2]);
  const Tensor k_lo = tensor(a[3]), k_hi = optional(a[4]), q_lo = optional(a[5]), q_hi = optional(a[6]), sinks_ = optional(a[7]);
  const float scale = real(a[8]);
  const bool grad = wants_gradient({q_, k_, v_, sinks_});
  Tensor q, k, v, sinks, o, lse;
  {
    at::NoGradGuard none;
    q = q_.contiguous();
    k = k_.contiguous();
    v = v_.contiguous();
    if (sinks_.defined()) sinks = sinks_.detach().to(at::kFloat).contiguous();
    if (grad)                                    // the backward pass's, before anything runs
      for (const Tensor& t : {q_lo, q_hi})
        operand(t, at::kInt, k.size(0), q, "first and last queries: an int32 for every key, on the keys' device");
    attn_forward(q, k, v, k_lo, k_hi, sinks, scale, o, lse);
  }
  if (grad) {
    auto node = make_node<AttnNode>({q_, k_, v_, sinks_});
    node->scale = scale;
    if (sinks_.defined()) {
      node->sink_type = sinks_.scalar_type();
      node->narrow_sinks = sinks_.scalar_type() == at::kBFloat16;
    }
    node->save({q, k, v, lse, k_lo, k_hi, q_lo, q_hi, sinks});
    torch::autograd::set_history(o, node);
    node->saved.emplace_back(o, true);
  }
  return tuple({o, lse});
  MCB_END
}

}  // namespace

#define MCB_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef autograd_methods[] = {MCB_FAST(linear), MCB_FAST(rmsnorm),   MCB_FAST(norm_linear), MCB_FAST(glu_linear),
                                  MCB_FAST(qkv),    MCB_FAST(attention), {nullptr, nullptr, 0, nullptr}};

}  // namespace mcb_host
