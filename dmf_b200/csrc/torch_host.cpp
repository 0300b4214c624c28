// Native host path of the Python surface: tensors in, one C++ call, kernels of libdmf_attn.so launched.
//
// What bounds it: nothing on the device.  A small attention call is a kernel of a few microseconds behind a Python
// route of 90 (torch custom op, ctypes structs, autograd.Function) to 480 us (under torch.func.jvp, where functorch
// builds a class for every custom_function_call, and where three of them follow one another for an adaLN block).  The
// functions below take the same steps natively:
//
//   * no functorch transform active: the op as a C++ autograd node (or the bare kernel when nothing needs a gradient);
//   * exactly one functorch JVP level (torch.func.jvp, how loss.py:165-170 reaches the ops): the inputs are unwrapped to
//     the tensors below that level, the op runs there - autograd at that level as usual - and primal and tangent are
//     wrapped again;
//   * anything else (tensor subclasses, dispatch modes, jit tracing, vmap / grad / nested transforms, arguments that the op
//     rejects, CPU tensors) returns None, and the Python caller takes the general route, which also raises the exact errors.
//
// What Python sees first (torch.compile, __torch_function__) is sorted out in _native.takes.
//
// Semantics are those of the autograd.Functions in flash_attn_jvp.py, rms_norm.py and adaln.py: tangents are plain
// inputs, backward differentiates the primal outputs only and once, tangent outputs carry no gradient (GELU, which stands in
// for a library function, excepted).
#include <ATen/ATen.h>
#include <ATen/FuncTorchTLS.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/functorch/DynamicLayer.h>
#include <ATen/functorch/TensorWrapper.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>
#include <optional>

#include "dmf_adaln.h"
#include "dmf_attn.h"
#include "dmf_step.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
namespace ft = at::functorch;

// ---- state shared with the Python module -----------------------------------------------------------------------------

constexpr int kMaxDevices = 64;
std::atomic<int64_t> g_launches{0};               // dmf_b200.ops.launch_count
std::atomic<int32_t*> g_status_word[kMaxDevices];  // device word kernels write to when a wait runs out (owned by Python)

// ---- which route ------------------------------------------------------------------------------------------------------

// A tensor this file handles itself: a plain CUDA tensor without Python dispatch, lazy conjugation / negation or an
// undefined-zero tangent behind it.
bool plain_cuda(const Tensor& t) {
  constexpr c10::DispatchKeySet odd({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot,
                                     c10::DispatchKey::ZeroTensor, c10::DispatchKey::Negative,
                                     c10::DispatchKey::Conjugate, c10::DispatchKey::Functionalize,
                                     c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::BatchedNestedTensor,
                                     c10::DispatchKey::Batched, c10::DispatchKey::FuncTorchGradWrapper});
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && (t.key_set() & odd).empty() && t.has_storage();
}

// Where the call stands: no transform, or one JVP level `level` whose wrappers are to be taken off and put on again.
struct Route {
  bool ok = false;
  bool jvp = false;
  int64_t level = 0;
};

Route find_route() {
  Route r;
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return r;
  if (torch::jit::tracer::isTracing()) return r;  // a trace has to see an op: a launch from here would leave no node in it
  const auto& stack = ft::getDynamicLayerStack();
  if (stack.empty()) {
    r.ok = true;
  } else if (stack.size() == 1 && stack[0].key() == ft::TransformType::Jvp) {
    r.ok = r.jvp = true;
    r.level = stack[0].layerId();
  }
  return r;
}

// Ops below the JVP level: functorch's two dispatch keys are what sends a call through the transform again, and its
// thread-local interpreter stack (the one level) is put aside, as C++ autograd nodes want to see none.
struct BelowTransform {
  explicit BelowTransform(bool on_) : on(on_) {
    if (!on) return;
    guard.emplace(c10::DispatchKeySet({c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                      c10::DispatchKey::FuncTorchDynamicLayerBackMode}));
    stack.swap(ft::functorchTLSAccessor());
  }
  ~BelowTransform() {
    if (on) stack.swap(ft::functorchTLSAccessor());
  }
  BelowTransform(const BelowTransform&) = delete;
  BelowTransform& operator=(const BelowTransform&) = delete;
  const bool on;
  std::optional<c10::impl::ExcludeDispatchKeyGuard> guard;
  std::unique_ptr<ft::FuncTorchTLSBase> stack;
};

// The tensor below the JVP level (the tensor itself if it is not one of that level's wrappers); undefined if unusable.
Tensor below(const Tensor& t, const Route& r) {
  if (!t.defined()) return t;
  if (r.jvp) {
    if (auto* w = ft::maybeGetTensorWrapper(t)) {
      if (!w->is_alive() || !w->level().has_value() || *w->level() != r.level) return Tensor();
      const Tensor inner = w->value();
      return plain_cuda(inner) ? inner : Tensor();
    }
  }
  return plain_cuda(t) ? t : Tensor();
}

// One input of an op: primal and (possibly undefined) tangent as tensors below the transform.
struct Dual {
  Tensor p, t;
};

bool split(const Tensor& x, const Route& r, Dual* out) {
  if (!x.defined()) return false;
  const Tensor& fw = x._fw_grad(0);
  if (fw.defined()) {
    out->t = below(fw, r);
    if (!out->t.defined()) return false;
  }
  out->p = below(x, r);
  if (!out->p.defined()) return false;
  if (r.jvp) {
    if (out->p._fw_grad(0).defined()) return false;  // a dual tensor of the level below as well: the general route
  } else if (fw.defined()) {
    out->p = out->p._fw_primal(0);
  }
  return true;
}

Tensor put_back(const Tensor& primal, const Tensor& tangent, const Route& r) {
  if (!r.jvp) {
    if (!tangent.defined()) return primal;
    return at::_make_dual(primal, tangent, 0);
  }
  Tensor w = ft::makeTensorWrapper(primal, r.level);
  if (tangent.defined()) w._set_fw_grad(ft::makeTensorWrapper(tangent, r.level), 0, /*is_inplace_op=*/false);
  return w;
}

// Optional inputs of an autograd node are std::optional: torch's C++ nodes take no undefined tensors.
std::optional<Tensor> maybe(const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; }
Tensor value_of(const std::optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }

bool needs_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// Gradients that a kernel's backward made cannot be differentiated again.  With create_graph they hang on this node, which
// raises when a second derivative is asked for - as the registered ops of the general route do - instead of leaving it out.
struct FirstOrderOnly : torch::autograd::Function<FirstOrderOnly> {
  static variable_list forward(AutogradContext*, at::TensorList grads, at::TensorList /*sources*/) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    variable_list out;
    for (const Tensor& g : grads) out.push_back(g.detach());
    return out;
  }
  static variable_list backward(AutogradContext*, variable_list) {
    TORCH_CHECK(false, "dmf_b200 ops have no second derivatives");
  }
};

// `grads` as a backward returns them, where they depend on `sources` (incoming gradient and saved tensors)
variable_list first_order_only(variable_list grads, std::initializer_list<const Tensor*> sources) {
  if (!needs_grad(sources)) return grads;
  variable_list made, from;
  for (const Tensor& g : grads)
    if (g.defined()) made.push_back(g);
  for (const Tensor* t : sources)
    if (t->defined() && t->requires_grad()) from.push_back(*t);
  const variable_list out = FirstOrderOnly::apply(at::TensorList(made), at::TensorList(from));
  auto next = out.begin();
  for (Tensor& g : grads)
    if (g.defined()) g = *next++;
  return grads;
}

// A gradient that is not a plain tensor (is_grads_batched, a subclass) goes to the registered op of the general route, which
// the dispatcher can unwrap.
template <typename R, typename... Args>
R registered_op(const char* name, const Args&... args) {
  const auto op = c10::Dispatcher::singleton().findSchemaOrThrow(name, "");
  return op.template typed<R(Args...)>().call(args...);
}

// ---- attention ----------------------------------------------------------------------------------------------------------

int attn_dtype(at::ScalarType t) {
  return t == at::kBFloat16 ? DMF_ATTN_BF16 : t == at::kHalf ? DMF_ATTN_FP16 : -1;
}

dmf_attn_tensor t4(const Tensor& x) { return {x.data_ptr(), x.stride(0), x.stride(1), x.stride(2)}; }

// slice i of a (B, L, 3, H, D) tensor
dmf_attn_tensor t4_packed(const Tensor& x, int i) {
  return {static_cast<char*>(x.data_ptr()) + i * x.stride(2) * static_cast<int64_t>(x.element_size()), x.stride(0), x.stride(1), x.stride(3)};
}

// the slices of a packed tensor can be read (and written) where they are
bool packed_ok(const Tensor& x) {
  return x.stride(4) == 1 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 && x.stride(0) % 8 == 0 && x.stride(1) % 8 == 0 &&
         x.stride(2) % 8 == 0 && x.stride(3) % 8 == 0;
}

// unit stride on D, 16-byte aligned base and strides (maybe_contiguous, models/flash_attention_2_jvp.py:24-25)
Tensor prep(const Tensor& x) {
  if (x.stride(3) == 1 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0) {
    bool ok = true;
    for (int i = 0; i < 3; ++i) ok = ok && x.stride(i) % 8 == 0;
    if (ok) return x;
  }
  return x.contiguous();
}

bool same_kind(const Tensor& a, const Tensor& b) {
  return b.dim() == 4 && a.scalar_type() == b.scalar_type() && a.device() == b.device();
}

// What ops.fwd_raw / fwd_dual_raw check; false: the general route raises the error.
bool attn_inputs_ok(const Tensor& q, const Tensor& k, const Tensor& v) {
  return q.dim() == 4 && attn_dtype(q.scalar_type()) >= 0 && same_kind(q, k) && same_kind(q, v) &&
         k.sizes() == v.sizes() && q.size(0) == k.size(0) && q.size(2) == k.size(2) && q.size(3) == k.size(3) &&
         g_status_word[q.get_device()].load(std::memory_order_acquire) != nullptr;
}

bool lse_ok(const Tensor& lse, const Tensor& o) {
  return lse.scalar_type() == at::kFloat && lse.device() == o.device() &&
         lse.sizes() == at::IntArrayRef({o.size(0), o.size(2), o.size(1)});
}

struct AttnOut {
  Tensor o, to, lse;
  int status = DMF_ATTN_OK;
};

template <typename A>
void attn_sizes(A* a, const Tensor& q, int64_t B, int64_t L, int64_t Lk, int64_t H, int64_t D, double scale) {
  a->batch = B; a->seqlen_q = L; a->seqlen_kv = Lk; a->heads = H; a->head_dim = D;
  a->dtype = attn_dtype(q.scalar_type());
  a->softmax_scale = static_cast<float>(scale);
  a->status_word = g_status_word[q.get_device()].load(std::memory_order_acquire);
  a->stream = c10::cuda::getCurrentCUDAStream(q.get_device()).stream();
}

// outputs and launch, with the inputs of `a` filled in
AttnOut attn_launch(dmf_attn_fwd_args* a, const Tensor& like, bool dual) {
  AttnOut r;
  const int64_t B = a->batch, L = a->seqlen_q, H = a->heads, D = a->head_dim;
  r.o = at::empty({B, L, H, D}, like.options());
  r.lse = at::empty({B, H, L}, like.options().dtype(at::kFloat));
  a->o = t4(r.o);
  a->lse = r.lse.data_ptr<float>();
  if (dual) {
    r.to = at::empty({B, L, H, D}, like.options());
    a->to = t4(r.to);
  }
  r.status = dual ? dmf_attn_fwd_dual(a) : dmf_attn_fwd(a);
  if (r.status == DMF_ATTN_OK) g_launches.fetch_add(1, std::memory_order_relaxed);
  return r;
}

AttnOut attn_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor* tq_, const Tensor* tk_,
                     const Tensor* tv_, double scale) {
  const c10::cuda::CUDAGuard device_guard(q_.device());
  const Tensor q = prep(q_), k = prep(k_), v = prep(v_);
  dmf_attn_fwd_args a = {};
  attn_sizes(&a, q, q.size(0), q.size(1), k.size(1), q.size(2), q.size(3), scale);
  a.q = t4(q); a.k = t4(k); a.v = t4(v);
  if (tq_ == nullptr) return attn_launch(&a, q, false);
  const Tensor tq = prep(*tq_), tk = prep(*tk_), tv = prep(*tv_);
  a.tq = t4(tq); a.tk = t4(tk); a.tv = t4(tv);
  return attn_launch(&a, q, true);
}

AttnOut attn_forward_packed(const Tensor& qkv_, const Tensor& tqkv_, double scale) {
  const c10::cuda::CUDAGuard device_guard(qkv_.device());
  const Tensor qkv = packed_ok(qkv_) ? qkv_ : qkv_.contiguous();
  dmf_attn_fwd_args a = {};
  attn_sizes(&a, qkv, qkv.size(0), qkv.size(1), qkv.size(1), qkv.size(3), qkv.size(4), scale);
  a.q = t4_packed(qkv, 0); a.k = t4_packed(qkv, 1); a.v = t4_packed(qkv, 2);
  if (!tqkv_.defined()) return attn_launch(&a, qkv, false);
  const Tensor t = packed_ok(tqkv_) ? tqkv_ : tqkv_.contiguous();
  a.tq = t4_packed(t, 0); a.tk = t4_packed(t, 1); a.tv = t4_packed(t, 2);
  return attn_launch(&a, qkv, true);
}

// Saved-tensor hooks hand back whatever they like: layouts are put right like those of inputs, anything else must be as saved.
void check_saved(bool as_saved) {
  TORCH_CHECK(as_saved, "dmf_b200 backward: a saved tensor came back with another type, shape or device");
}

// workspace and launch of a backward, with the tensors of `a` filled in
void attn_launch_bwd(dmf_attn_bwd_args* a, const Tensor& like, const Tensor& lse) {
  const size_t bytes = dmf_attn_bwd_workspace_bytes(a->batch, a->seqlen_q, a->seqlen_kv, a->heads, a->head_dim);
  const Tensor ws = at::empty({static_cast<int64_t>(std::max<size_t>(bytes, 16))}, like.options().dtype(at::kByte));
  a->lse = lse.data_ptr<float>();
  a->workspace = ws.data_ptr();
  a->workspace_bytes = bytes;
  const int st = dmf_attn_bwd(a);
  TORCH_CHECK(st == DMF_ATTN_OK, "dmf_attn: ", dmf_attn_status_string(st));
  g_launches.fetch_add(2, std::memory_order_relaxed);
}

variable_list attn_backward(const Tensor& dout_, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& o_,
                            const Tensor& lse_, double scale) {
  for (const Tensor* t : {&q_, &k_, &v_, &o_, &lse_}) check_saved(plain_cuda(*t));
  check_saved(attn_inputs_ok(q_, k_, v_) && same_kind(q_, o_) && o_.sizes() == q_.sizes() && lse_ok(lse_, o_));
  const c10::cuda::CUDAGuard device_guard(q_.device());
  TORCH_CHECK(same_kind(q_, dout_) && dout_.sizes() == o_.sizes(), "dmf_b200 attention backward: unexpected gradient");
  const Tensor dout = prep(dout_), q = prep(q_), k = prep(k_), v = prep(v_), o = prep(o_), lse = lse_.contiguous();
  variable_list grads = {at::empty(q.sizes(), q.options()), at::empty(k.sizes(), q.options()), at::empty(v.sizes(), q.options())};
  dmf_attn_bwd_args a = {};
  attn_sizes(&a, q, q.size(0), q.size(1), k.size(1), q.size(2), q.size(3), scale);
  a.dout = t4(dout); a.q = t4(q); a.k = t4(k); a.v = t4(v); a.o = t4(o);
  a.dq = t4(grads[0]); a.dk = t4(grads[1]); a.dv = t4(grads[2]);
  attn_launch_bwd(&a, q, lse);
  return grads;
}

// one (B, L, 3, H, D) gradient
Tensor attn_backward_packed(const Tensor& dout_, const Tensor& qkv_, const Tensor& o_, const Tensor& lse_, double scale) {
  for (const Tensor* t : {&qkv_, &o_, &lse_}) check_saved(plain_cuda(*t));
  check_saved(qkv_.dim() == 5 && qkv_.size(2) == 3 && attn_dtype(qkv_.scalar_type()) >= 0 &&
              o_.scalar_type() == qkv_.scalar_type() && o_.device() == qkv_.device() &&
              o_.sizes() == at::IntArrayRef({qkv_.size(0), qkv_.size(1), qkv_.size(3), qkv_.size(4)}) && lse_ok(lse_, o_));
  const c10::cuda::CUDAGuard device_guard(qkv_.device());
  TORCH_CHECK(dout_.scalar_type() == o_.scalar_type() && dout_.device() == o_.device() && dout_.sizes() == o_.sizes(),
              "dmf_b200 attention backward: unexpected gradient");
  const Tensor dout = prep(dout_), o = prep(o_), lse = lse_.contiguous(), qkv = packed_ok(qkv_) ? qkv_ : qkv_.contiguous();
  const Tensor grad = at::empty(qkv.sizes(), qkv.options());
  dmf_attn_bwd_args a = {};
  attn_sizes(&a, qkv, qkv.size(0), qkv.size(1), qkv.size(1), qkv.size(3), qkv.size(4), scale);
  a.dout = t4(dout); a.o = t4(o);
  a.q = t4_packed(qkv, 0); a.k = t4_packed(qkv, 1); a.v = t4_packed(qkv, 2);
  a.dq = t4_packed(grad, 0); a.dk = t4_packed(grad, 1); a.dv = t4_packed(grad, 2);
  attn_launch_bwd(&a, qkv, lse);
  return grad;
}

struct RejectedError : std::exception {};  // the C ABI refused before any launch: the general route reports it

struct AttnNode : torch::autograd::Function<AttnNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                               const std::optional<Tensor>& tq, const std::optional<Tensor>& tk,
                               const std::optional<Tensor>& tv, double scale) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    const bool dual = tq.has_value();
    AttnOut r = attn_forward(q, k, v, dual ? &*tq : nullptr, dual ? &*tk : nullptr, dual ? &*tv : nullptr, scale);
    if (r.status != DMF_ATTN_OK) throw RejectedError();
    ctx->save_for_backward({q, k, v, r.o, r.lse});
    ctx->saved_data["scale"] = scale;
    ctx->set_materialize_grads(false);
    return dual ? variable_list{r.o, r.to} : variable_list{r.o};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    if (grads[0].defined() && !plain_cuda(grads[0])) {
      const auto [dq, dk, dv] = registered_op<std::tuple<Tensor, Tensor, Tensor>>(
          "dmf_b200::attn_bwd", grads[0], s[0], s[1], s[2], s[3], s[4], ctx->saved_data["scale"].toDouble());
      return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor()};
    }
    variable_list g = backward_once(ctx, grads, s);
    g.resize(7);
    return first_order_only(std::move(g), {&grads[0], &s[0], &s[1], &s[2]});
  }
  static variable_list backward_once(AutogradContext* ctx, const variable_list& grads, const variable_list& s) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    if (!grads[0].defined())  // only the tangent output was used: it carries no gradient
      return {at::zeros_like(s[0]), at::zeros_like(s[1]), at::zeros_like(s[2])};
    return attn_backward(grads[0], s[0], s[1], s[2], s[3], s[4], ctx->saved_data["scale"].toDouble());
  }
};

struct AttnPackedNode : torch::autograd::Function<AttnPackedNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& qkv, const std::optional<Tensor>& tqkv, double scale) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    AttnOut r = attn_forward_packed(qkv, value_of(tqkv), scale);
    if (r.status != DMF_ATTN_OK) throw RejectedError();
    ctx->save_for_backward({qkv, r.o, r.lse});
    ctx->saved_data["scale"] = scale;
    ctx->set_materialize_grads(false);
    return r.to.defined() ? variable_list{r.o, r.to} : variable_list{r.o};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    if (grads[0].defined() && !plain_cuda(grads[0]))
      return {registered_op<Tensor>("dmf_b200::attn_bwd_qkvpacked", grads[0], s[0], s[1], s[2],
                                    ctx->saved_data["scale"].toDouble()), Tensor(), Tensor()};
    return first_order_only({backward_once(ctx, grads, s), Tensor(), Tensor()}, {&grads[0], &s[0]});
  }
  static Tensor backward_once(AutogradContext* ctx, const variable_list& grads, const variable_list& s) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    if (!grads[0].defined()) return at::zeros_like(s[0]);
    return attn_backward_packed(grads[0], s[0], s[1], s[2], ctx->saved_data["scale"].toDouble());
  }
};

std::optional<Tensor> attn_func(const Tensor& q_, const Tensor& k_, const Tensor& v_, std::optional<double> softmax_scale) {
  const Route route = find_route();
  Dual q, k, v;
  if (!route.ok || !split(q_, route, &q) || !split(k_, route, &k) || !split(v_, route, &v)) return std::nullopt;
  if (!attn_inputs_ok(q.p, k.p, v.p)) return std::nullopt;
  const bool dual = q.t.defined() || k.t.defined() || v.t.defined();
  std::optional<BelowTransform> guard(std::in_place, route.jvp);
  if (dual)
    for (Dual* d : {&q, &k, &v}) {
      if (!d->t.defined()) d->t = at::zeros_like(d->p);
      if (d->t.sizes() != d->p.sizes() || !same_kind(q.p, d->t)) return std::nullopt;
    }
  const double scale = softmax_scale.has_value() ? *softmax_scale : std::pow(static_cast<double>(q.p.size(3)), -0.5);
  Tensor o, to;
  if (needs_grad({&q.p, &k.p, &v.p, &q.t, &k.t, &v.t})) {
    try {
      variable_list out = AttnNode::apply(q.p, k.p, v.p, maybe(q.t), maybe(k.t), maybe(v.t), scale);
      o = out[0];
      if (dual) to = out[1];
    } catch (const RejectedError&) {
      return std::nullopt;
    }
  } else {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    AttnOut r = attn_forward(q.p, k.p, v.p, dual ? &q.t : nullptr, dual ? &k.t : nullptr, dual ? &v.t : nullptr, scale);
    if (r.status != DMF_ATTN_OK) return std::nullopt;
    o = r.o;
    to = r.to;
  }
  guard.reset();
  return put_back(o, to, route);
}

std::optional<Tensor> attn_qkvpacked(const Tensor& qkv_, std::optional<double> softmax_scale) {
  const Route route = find_route();
  Dual x;
  if (!route.ok || !split(qkv_, route, &x)) return std::nullopt;
  if (x.p.dim() != 5 || x.p.size(2) != 3 || attn_dtype(x.p.scalar_type()) < 0 ||
      g_status_word[x.p.get_device()].load(std::memory_order_acquire) == nullptr)
    return std::nullopt;
  const bool dual = x.t.defined();
  if (dual && (x.t.sizes() != x.p.sizes() || x.t.scalar_type() != x.p.scalar_type() || x.t.device() != x.p.device()))
    return std::nullopt;
  std::optional<BelowTransform> guard(std::in_place, route.jvp);
  const double scale = softmax_scale.has_value() ? *softmax_scale : std::pow(static_cast<double>(x.p.size(4)), -0.5);
  Tensor o, to;
  if (needs_grad({&x.p, &x.t})) {
    try {
      variable_list out = AttnPackedNode::apply(x.p, maybe(x.t), scale);
      o = out[0];
      if (dual) to = out[1];
    } catch (const RejectedError&) {
      return std::nullopt;
    }
  } else {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    AttnOut r = attn_forward_packed(x.p, x.t, scale);
    if (r.status != DMF_ATTN_OK) return std::nullopt;
    o = r.o;
    to = r.to;
  }
  guard.reset();
  return put_back(o, to, route);
}

// ---- per-head RMS norm -----------------------------------------------------------------------------------------------

// the weight as the kernel reads it: in the tensors' own 16-bit type where it is there already, else fp32
Tensor rms_weight(const Tensor& w, const Tensor& x) {
  const Tensor d = w.detach();
  if (d.scalar_type() == x.scalar_type() && d.device() == x.device() && d.is_contiguous() &&
      reinterpret_cast<uintptr_t>(d.data_ptr()) % 16 == 0)
    return d;
  if (d.scalar_type() == at::kFloat && d.device() == x.device() && d.is_contiguous()) return d;
  return d.to(x.options().dtype(at::kFloat)).contiguous();
}

int rms_dtype(const Tensor& x, const Tensor& w) {
  return attn_dtype(x.scalar_type()) + (w.scalar_type() == at::kFloat ? 0 : DMF_RMSNORM_WEIGHT_16BIT);
}

struct PairOut {
  Tensor y, ty;
  int status = DMF_ATTN_OK;
};

PairOut rms_forward(const Tensor& x_, const Tensor& tx_, const Tensor& weight, double eps) {
  const c10::cuda::CUDAGuard device_guard(x_.device());
  const Tensor x = prep(x_), w = rms_weight(weight, x);
  PairOut r;
  r.y = at::empty(x.sizes(), x.options());
  dmf_rmsnorm_args a = {};
  a.batch = x.size(0); a.seqlen = x.size(1); a.heads = x.size(2); a.head_dim = x.size(3);
  a.dtype = rms_dtype(x, w);
  a.eps = static_cast<float>(eps);
  a.x = t4(x); a.y = t4(r.y);
  Tensor tx;
  if (tx_.defined()) {
    tx = prep(tx_);
    r.ty = at::empty(x.sizes(), x.options());
    a.tx = t4(tx); a.ty = t4(r.ty);
  }
  a.weight = w.data_ptr();
  a.stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
  r.status = w.numel() == x.size(3) ? dmf_rmsnorm_fwd(&a) : static_cast<int>(DMF_ATTN_ERR_SHAPE);
  if (r.status == DMF_ATTN_OK) g_launches.fetch_add(1, std::memory_order_relaxed);
  return r;
}

struct RmsNode : torch::autograd::Function<RmsNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& tx, const Tensor& weight,
                               double eps) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = rms_forward(x, value_of(tx), weight, eps);
    if (r.status != DMF_ATTN_OK) throw RejectedError();
    ctx->save_for_backward({x, weight});
    ctx->saved_data["eps"] = eps;
    ctx->set_materialize_grads(false);
    return r.ty.defined() ? variable_list{r.y, r.ty} : variable_list{r.y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    if (grads[0].defined() && !plain_cuda(grads[0])) {
      const auto [dx, dw] = registered_op<std::tuple<Tensor, Tensor>>("dmf_b200::rmsnorm_bwd", grads[0], s[0], s[1],
                                                                      ctx->saved_data["eps"].toDouble());
      return {dx, Tensor(), dw.to(s[1].scalar_type()), Tensor()};
    }
    return first_order_only(backward_once(ctx, grads, s), {&grads[0], &s[0], &s[1]});
  }
  static variable_list backward_once(AutogradContext* ctx, const variable_list& grads, const variable_list& s) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    if (!grads[0].defined()) return {at::zeros_like(s[0]), Tensor(), at::zeros_like(s[1]), Tensor()};
    check_saved(plain_cuda(s[0]) && s[0].dim() == 4 && attn_dtype(s[0].scalar_type()) >= 0 && s[1].numel() == s[0].size(3));
    const c10::cuda::CUDAGuard device_guard(s[0].device());
    TORCH_CHECK(same_kind(s[0], grads[0]) && s[0].sizes() == grads[0].sizes(), "dmf_b200 RMS norm backward: unexpected gradient");
    const Tensor x = prep(s[0]), dy = prep(grads[0]), w = rms_weight(s[1], x);
    const int64_t D = x.size(3);
    const Tensor dx = at::empty(x.sizes(), x.options());
    const Tensor dw = at::empty({D}, x.options().dtype(at::kFloat));
    const size_t bytes = dmf_rmsnorm_bwd_workspace_bytes(D);
    const Tensor ws = at::empty({static_cast<int64_t>(bytes)}, x.options().dtype(at::kByte));
    dmf_rmsnorm_bwd_args a = {};
    a.batch = x.size(0); a.seqlen = x.size(1); a.heads = x.size(2); a.head_dim = D;
    a.dtype = rms_dtype(x, w);
    a.eps = static_cast<float>(ctx->saved_data["eps"].toDouble());
    a.dy = t4(dy); a.x = t4(x); a.dx = t4(dx);
    a.weight = w.data_ptr();
    a.dweight = dw.data_ptr<float>();
    a.workspace = ws.data_ptr();
    a.workspace_bytes = bytes;
    a.stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
    const int st = dmf_rmsnorm_bwd(&a);
    TORCH_CHECK(st == DMF_ATTN_OK, "dmf_attn: ", dmf_attn_status_string(st));
    g_launches.fetch_add(2, std::memory_order_relaxed);
    return {dx, Tensor(), dw.to(s[1].scalar_type()), Tensor()};
  }
};

std::optional<Tensor> rms_norm(const Tensor& x_, const Tensor& weight_, double eps) {
  const Route route = find_route();
  Dual x, w;
  if (!route.ok || !split(x_, route, &x) || !split(weight_, route, &w)) return std::nullopt;
  if (x.p.dim() != 4 || attn_dtype(x.p.scalar_type()) < 0) return std::nullopt;
  if (x.t.defined() && (x.t.sizes() != x.p.sizes() || !same_kind(x.p, x.t))) return std::nullopt;
  std::optional<BelowTransform> guard(std::in_place, route.jvp);
  Tensor y, ty;
  if (needs_grad({&x.p, &x.t, &w.p})) {
    try {
      variable_list out = RmsNode::apply(x.p, maybe(x.t), w.p, eps);
      y = out[0];
      if (x.t.defined()) ty = out[1];
    } catch (const RejectedError&) {
      return std::nullopt;
    }
  } else {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = rms_forward(x.p, x.t, w.p, eps);
    if (r.status != DMF_ATTN_OK) return std::nullopt;
    y = r.y;
    ty = r.ty;
  }
  guard.reset();
  return put_back(y, ty, route);
}

// ---- adaLN ops -----------------------------------------------------------------------------------------------------------

int ada_dtype(at::ScalarType t) { return t == at::kFloat ? DMF_ADALN_F32 : t == at::kBFloat16 ? DMF_ADALN_BF16 : -1; }

bool ada_pair_ok(at::ScalarType wide, at::ScalarType narrow) {
  return (wide == at::kFloat && (narrow == at::kFloat || narrow == at::kBFloat16)) ||
         (wide == at::kBFloat16 && narrow == at::kBFloat16);
}

// rows read as 4-element vectors: unit channel stride, 16-byte aligned base, row strides that are multiples of 4 elements
Tensor ada_rows(const Tensor& t) {
  if (t.stride(2) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && t.stride(0) % 4 == 0 && t.stride(1) % 4 == 0)
    return t;
  return t.contiguous();
}

bool ada_mod_fits(const Tensor& t, const Tensor& x) {
  if (!t.defined()) return true;
  if (ada_dtype(t.scalar_type()) < 0 || t.device() != x.device()) return false;
  const int64_t d = t.dim();
  return (d == 2 || (d == 3 && t.size(1) == 1)) && t.size(0) == x.size(0) && t.size(d - 1) == x.size(2);
}

// a (B, C) or (B, 1, C) modulation tensor as a 2-D one with unit channel stride
Tensor ada_mod(const Tensor& t_, at::ScalarType dtype) {
  if (!t_.defined()) return t_;
  Tensor t = t_.dim() == 3 ? t_.select(1, 0) : t_;
  if (t.scalar_type() != dtype) t = t.to(dtype);
  if (t.stride(1) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0 || t.stride(0) % 4 != 0) t = t.contiguous();
  return t;
}

at::ScalarType ada_mod_dtype(std::initializer_list<const Tensor*> mods) {
  for (const Tensor* m : mods)
    if (m->defined() && m->scalar_type() == at::kFloat) return at::kFloat;
  return at::kBFloat16;
}

dmf_rows ada_r(const Tensor& t) { return t.defined() ? dmf_rows{t.data_ptr(), t.stride(0), t.stride(1)} : dmf_rows{}; }
dmf_mod ada_m(const Tensor& t) { return t.defined() ? dmf_mod{t.data_ptr(), t.stride(0)} : dmf_mod{}; }

template <typename A>
void ada_head(A* a, const Tensor& x, at::ScalarType narrow, at::ScalarType mod) {
  a->batch = x.size(0); a->seqlen = x.size(1); a->channels = x.size(2);
  a->wide_dtype = ada_dtype(x.scalar_type());
  a->narrow_dtype = ada_dtype(narrow);
  a->mod_dtype = ada_dtype(mod);
  a->stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
}

PairOut ln_forward(const Tensor& x_, const Tensor& tx_, const Tensor& shift_, const Tensor& scale_, const Tensor& tshift_,
                   const Tensor& tscale_, double eps, at::ScalarType out_dtype) {
  const c10::cuda::CUDAGuard device_guard(x_.device());
  const at::ScalarType md = ada_mod_dtype({&shift_, &scale_, &tshift_, &tscale_});
  const Tensor x = ada_rows(x_), shift = ada_mod(shift_, md), scale = ada_mod(scale_, md);
  Tensor tx, tshift, tscale;
  if (tx_.defined()) {
    tx = ada_rows(tx_.scalar_type() == x.scalar_type() ? tx_ : tx_.to(x.scalar_type()));
    if (tshift_.defined() || tscale_.defined()) {  // the kernel takes the two modulation tangents together
      tshift = tshift_.defined() ? ada_mod(tshift_, md) : at::zeros_like(shift);
      tscale = tscale_.defined() ? ada_mod(tscale_, md) : at::zeros_like(scale);
    }
  }
  PairOut r;
  const auto narrow = x.options().dtype(out_dtype);
  r.y = at::empty(x.sizes(), narrow);
  if (tx.defined()) r.ty = at::empty(x.sizes(), narrow);
  dmf_ln_modulate_args a = {};
  ada_head(&a, x, out_dtype, md);
  a.eps = static_cast<float>(eps);
  a.x = ada_r(x); a.tx = ada_r(tx); a.y = ada_r(r.y); a.ty = ada_r(r.ty);
  a.shift = ada_m(shift); a.scale = ada_m(scale); a.tshift = ada_m(tshift); a.tscale = ada_m(tscale);
  r.status = dmf_ln_modulate_fwd(&a);
  if (r.status == DMF_ATTN_OK) g_launches.fetch_add(1, std::memory_order_relaxed);
  return r;
}

Tensor ada_workspace(const Tensor& x, size_t* bytes) {
  *bytes = dmf_adaln_bwd_workspace_bytes(x.size(0), x.size(1), x.size(2));
  return at::empty({static_cast<int64_t>(*bytes)}, x.options().dtype(at::kByte));
}

// a (B, C) fp32 gradient in the shape and type of its modulation tensor
Tensor ada_mod_grad(const Tensor& g, const Tensor& like) { return g.to(like.scalar_type()).reshape(like.sizes()); }

struct LnNode : torch::autograd::Function<LnNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& tx, const Tensor& shift,
                               const Tensor& scale, const std::optional<Tensor>& tshift, const std::optional<Tensor>& tscale,
                               double eps, int64_t out_dtype) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = ln_forward(x, value_of(tx), shift, scale, value_of(tshift), value_of(tscale), eps,
                           static_cast<at::ScalarType>(out_dtype));
    if (r.status != DMF_ATTN_OK) throw RejectedError();
    ctx->save_for_backward({x, scale});
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["shift_shape"] = shift.sizes().vec();
    ctx->saved_data["shift_dtype"] = static_cast<int64_t>(shift.scalar_type());
    ctx->set_materialize_grads(false);
    return r.ty.defined() ? variable_list{r.y, r.ty} : variable_list{r.y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    return first_order_only(backward_once(ctx, grads, s), {&grads[0], &s[0], &s[1]});
  }
  static variable_list backward_once(AutogradContext* ctx, const variable_list& grads, const variable_list& s) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    const auto shift_shape = ctx->saved_data["shift_shape"].toIntVector();
    const auto shift_dtype = static_cast<at::ScalarType>(ctx->saved_data["shift_dtype"].toInt());
    if (!grads[0].defined())
      return {at::zeros_like(s[0]), Tensor(), at::zeros(shift_shape, s[1].options().dtype(shift_dtype)),
              at::zeros_like(s[1]), Tensor(), Tensor(), Tensor(), Tensor()};
    check_saved(plain_cuda(s[0]) && plain_cuda(s[1]) && s[0].dim() == 3 && ada_mod_fits(s[1], s[0]));
    const c10::cuda::CUDAGuard device_guard(s[0].device());
    TORCH_CHECK(plain_cuda(grads[0]), "dmf_b200 LayerNorm-modulate backward: unexpected gradient");
    const Tensor x = ada_rows(s[0]), dy = ada_rows(grads[0]);
    TORCH_CHECK(dy.sizes() == x.sizes() && ada_pair_ok(x.scalar_type(), dy.scalar_type()),
                "dmf_b200 LayerNorm-modulate backward: unexpected gradient");
    const at::ScalarType md = ada_mod_dtype({&s[1]});
    const Tensor scale = ada_mod(s[1], md);
    const Tensor dx = at::empty(x.sizes(), x.options());
    const Tensor dmod = at::empty({2, x.size(0), x.size(2)}, x.options().dtype(at::kFloat));
    dmf_ln_modulate_bwd_args a = {};
    const Tensor ws = ada_workspace(x, &a.workspace_bytes);
    ada_head(&a, x, dy.scalar_type(), md);
    a.eps = static_cast<float>(ctx->saved_data["eps"].toDouble());
    a.dy = ada_r(dy); a.x = ada_r(x); a.dx = ada_r(dx); a.scale = ada_m(scale);
    a.dshift = dmod.data_ptr<float>();
    a.dscale = a.dshift + x.size(0) * x.size(2);
    a.workspace = ws.data_ptr();
    const int st = dmf_ln_modulate_bwd(&a);
    TORCH_CHECK(st == DMF_ATTN_OK, "dmf_attn: ", dmf_attn_status_string(st));
    g_launches.fetch_add(2, std::memory_order_relaxed);
    const Tensor dshift = dmod.select(0, 0).to(shift_dtype).reshape(shift_shape);
    return {dx, Tensor(), dshift, ada_mod_grad(dmod.select(0, 1), s[1]), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

std::optional<Tensor> ln_modulate(const Tensor& x_, const Tensor& shift_, const Tensor& scale_, double eps,
                                  std::optional<at::ScalarType> out_dtype) {
  const Route route = find_route();
  Dual x, shift, scale;
  if (!route.ok || !split(x_, route, &x) || !split(shift_, route, &shift) || !split(scale_, route, &scale)) return std::nullopt;
  const at::ScalarType narrow = out_dtype.has_value() ? *out_dtype
                                : at::autocast::is_autocast_enabled(at::kCUDA) ? at::autocast::get_autocast_dtype(at::kCUDA)
                                                                               : x.p.scalar_type();
  if (x.p.dim() != 3 || !ada_pair_ok(x.p.scalar_type(), narrow)) return std::nullopt;
  for (const Tensor* m : {&shift.p, &shift.t, &scale.p, &scale.t})
    if (!ada_mod_fits(*m, x.p)) return std::nullopt;
  const bool dual = x.t.defined() || shift.t.defined() || scale.t.defined();
  std::optional<BelowTransform> guard(std::in_place, route.jvp);
  if (dual && !x.t.defined()) x.t = at::zeros_like(x.p);
  if (dual && x.t.sizes() != x.p.sizes()) return std::nullopt;
  Tensor y, ty;
  if (needs_grad({&x.p, &shift.p, &scale.p, &x.t, &shift.t, &scale.t})) {
    try {
      variable_list out = LnNode::apply(x.p, maybe(x.t), shift.p, scale.p, maybe(shift.t), maybe(scale.t), eps,
                                        static_cast<int64_t>(narrow));
      y = out[0];
      if (dual) ty = out[1];
    } catch (const RejectedError&) {
      return std::nullopt;
    }
  } else {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = ln_forward(x.p, x.t, shift.p, scale.p, shift.t, scale.t, eps, narrow);
    if (r.status != DMF_ATTN_OK) return std::nullopt;
    y = r.y;
    ty = r.ty;
  }
  guard.reset();
  return put_back(y, ty, route);
}

PairOut gate_forward(const Tensor& x_, const Tensor& tx_, const Tensor& h_, const Tensor& th_, const Tensor& gate_,
                     const Tensor& tgate_) {
  const c10::cuda::CUDAGuard device_guard(x_.device());
  const at::ScalarType md = ada_mod_dtype({&gate_, &tgate_});
  const Tensor x = ada_rows(x_), h = ada_rows(h_), gate = ada_mod(gate_, md);
  Tensor tx, th, tgate;
  if (tx_.defined() || th_.defined() || tgate_.defined()) {
    tx = tx_.defined() ? ada_rows(tx_.scalar_type() == x.scalar_type() ? tx_ : tx_.to(x.scalar_type())) : at::zeros_like(x);
    th = th_.defined() ? ada_rows(th_.scalar_type() == h.scalar_type() ? th_ : th_.to(h.scalar_type())) : at::zeros_like(h);
    tgate = ada_mod(tgate_, md);
  }
  PairOut r;
  r.y = at::empty(x.sizes(), x.options());
  if (tx.defined()) r.ty = at::empty(x.sizes(), x.options());
  dmf_gate_residual_args a = {};
  ada_head(&a, x, h.scalar_type(), md);
  a.x = ada_r(x); a.tx = ada_r(tx); a.h = ada_r(h); a.th = ada_r(th); a.out = ada_r(r.y); a.tout = ada_r(r.ty);
  a.gate = ada_m(gate); a.tgate = ada_m(tgate);
  r.status = dmf_gate_residual_fwd(&a);
  if (r.status == DMF_ATTN_OK) g_launches.fetch_add(1, std::memory_order_relaxed);
  return r;
}

struct GateNode : torch::autograd::Function<GateNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& tx, const Tensor& h,
                               const std::optional<Tensor>& th, const Tensor& gate, const std::optional<Tensor>& tgate) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = gate_forward(x, value_of(tx), h, value_of(th), gate, value_of(tgate));
    if (r.status != DMF_ATTN_OK) throw RejectedError();
    ctx->save_for_backward({h, gate});
    ctx->saved_data["x_dtype"] = static_cast<int64_t>(x.scalar_type());
    ctx->set_materialize_grads(false);
    return r.ty.defined() ? variable_list{r.y, r.ty} : variable_list{r.y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    variable_list g = first_order_only(backward_once(ctx, grads, s), {&grads[0], &s[0], &s[1]});
    if (grads[0].defined()) g[0] = grads[0];  // x's gradient is the incoming one, with its graph
    return g;
  }
  // all but x's gradient, which is the incoming one (zero where only the tangent output was used)
  static variable_list backward_once(AutogradContext* ctx, const variable_list& grads, const variable_list& s) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    if (!grads[0].defined())
      return {at::zeros_like(s[0], at::TensorOptions().dtype(static_cast<at::ScalarType>(ctx->saved_data["x_dtype"].toInt()))),
              Tensor(), at::zeros_like(s[0]), Tensor(), at::zeros_like(s[1]), Tensor()};
    check_saved(plain_cuda(s[0]) && plain_cuda(s[1]) && s[0].dim() == 3 && ada_mod_fits(s[1], s[0]));
    const c10::cuda::CUDAGuard device_guard(s[0].device());
    TORCH_CHECK(plain_cuda(grads[0]), "dmf_b200 gate-residual backward: unexpected gradient");
    const Tensor dout = ada_rows(grads[0]), h = ada_rows(s[0]);
    TORCH_CHECK(dout.sizes() == h.sizes() && ada_pair_ok(dout.scalar_type(), h.scalar_type()),
                "dmf_b200 gate-residual backward: unexpected gradient");
    const at::ScalarType md = ada_mod_dtype({&s[1]});
    const Tensor gate = ada_mod(s[1], md);
    const Tensor dh = at::empty(h.sizes(), h.options());
    const Tensor dgate = at::empty({h.size(0), h.size(2)}, h.options().dtype(at::kFloat));
    dmf_gate_residual_bwd_args a = {};
    const Tensor ws = ada_workspace(h, &a.workspace_bytes);
    ada_head(&a, dout, h.scalar_type(), md);
    a.dout = ada_r(dout); a.h = ada_r(h); a.dh = ada_r(dh); a.gate = ada_m(gate);
    a.dgate = dgate.data_ptr<float>();
    a.workspace = ws.data_ptr();
    const int st = dmf_gate_residual_bwd(&a);
    TORCH_CHECK(st == DMF_ATTN_OK, "dmf_attn: ", dmf_attn_status_string(st));
    g_launches.fetch_add(2, std::memory_order_relaxed);
    return {Tensor(), Tensor(), dh, Tensor(), ada_mod_grad(dgate, s[1]), Tensor()};
  }
};

std::optional<Tensor> gate_residual(const Tensor& x_, const Tensor& gate_, const Tensor& h_) {
  const Route route = find_route();
  Dual x, h, gate;
  if (!route.ok || !split(x_, route, &x) || !split(h_, route, &h) || !split(gate_, route, &gate)) return std::nullopt;
  if (x.p.dim() != 3 || h.p.sizes() != x.p.sizes() || h.p.device() != x.p.device() ||
      !ada_pair_ok(x.p.scalar_type(), h.p.scalar_type()))
    return std::nullopt;
  for (const Tensor* t : {&x.t, &h.t})
    if (t->defined() && t->sizes() != x.p.sizes()) return std::nullopt;
  for (const Tensor* m : {&gate.p, &gate.t})
    if (!ada_mod_fits(*m, x.p)) return std::nullopt;
  std::optional<BelowTransform> guard(std::in_place, route.jvp);
  Tensor y, ty;
  if (needs_grad({&x.p, &h.p, &gate.p, &x.t, &h.t, &gate.t})) {
    try {
      variable_list out = GateNode::apply(x.p, maybe(x.t), h.p, maybe(h.t), gate.p, maybe(gate.t));
      y = out[0];
      if (out.size() > 1) ty = out[1];
    } catch (const RejectedError&) {
      return std::nullopt;
    }
  } else {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = gate_forward(x.p, x.t, h.p, h.t, gate.p, gate.t);
    if (r.status != DMF_ATTN_OK) return std::nullopt;
    y = r.y;
    ty = r.ty;
  }
  guard.reset();
  return put_back(y, ty, route);
}

// ---- GELU ----------------------------------------------------------------------------------------------------------------

// one flat run of elements the kernel reads as 16-byte vectors
Tensor gelu_flat(const Tensor& t) {
  const Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0 ? c : c.clone();
}

int gelu_launch(const Tensor& x, const Tensor& t, const Tensor& y, const Tensor& ty) {
  dmf_gelu_args a = {};
  a.count = x.numel();
  a.dtype = attn_dtype(x.scalar_type());
  a.x = x.data_ptr();
  if (t.defined()) a.t = t.data_ptr();
  if (y.defined()) a.y = y.data_ptr();
  if (ty.defined()) a.ty = ty.data_ptr();
  a.stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
  return dmf_gelu(&a);  // not in g_launches, which counts the attention, norm and adaLN kernels
}

PairOut gelu_forward(const Tensor& x_, const Tensor& tx_) {
  const c10::cuda::CUDAGuard device_guard(x_.device());
  const Tensor x = gelu_flat(x_);
  PairOut r;
  r.y = at::empty(x.sizes(), x.options());
  Tensor tx;
  if (tx_.defined()) {
    tx = gelu_flat(tx_);
    r.ty = at::empty(x.sizes(), x.options());
  }
  r.status = gelu_launch(x, tx, r.y, r.ty);
  return r;
}

// gelu'(x) dy by the kernel
Tensor gelu_gradient(const Tensor& x_, const Tensor& dy_) {
  check_saved(plain_cuda(x_) && attn_dtype(x_.scalar_type()) >= 0);
  const c10::cuda::CUDAGuard device_guard(x_.device());
  TORCH_CHECK(dy_.sizes() == x_.sizes() && dy_.scalar_type() == x_.scalar_type() && dy_.device() == x_.device(),
              "dmf_b200 GELU backward: unexpected gradient");
  const Tensor x = gelu_flat(x_), dy = gelu_flat(dy_);
  const Tensor dx = at::empty(x.sizes(), x.options());
  const int st = gelu_launch(x, dy, Tensor(), dx);
  TORCH_CHECK(st == DMF_ATTN_OK, "dmf_attn: ", dmf_attn_status_string(st));
  return dx;
}

// Unlike the other ops' nodes this one differentiates its tangent output too, as the library's GELU does: rarely wanted
// (a loss that does not detach the tangent), and left to differentiable library calls.
struct GeluNode : torch::autograd::Function<GeluNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& tx) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = gelu_forward(x, value_of(tx));
    if (r.status != DMF_ATTN_OK) throw RejectedError();
    ctx->save_for_backward(tx.has_value() ? variable_list{x, *tx} : variable_list{x});
    ctx->set_materialize_grads(false);
    return r.ty.defined() ? variable_list{r.y, r.ty} : variable_list{r.y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    Tensor dx, dtx;
    if (grads[0].defined()) {
      if (needs_grad({&grads[0], &s[0]}) || !plain_cuda(grads[0])) {
        dx = at::gelu_backward(grads[0], s[0], "tanh");  // differentiable again, and for batched gradients
      } else {
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        dx = gelu_gradient(s[0], grads[0]);
      }
    }
    if (grads.size() > 1 && grads[1].defined()) {  // ty = gelu'(x) tx
      const bool create_graph = at::GradMode::is_enabled();
      const at::AutoGradMode with_graph(true);
      const Tensor x = create_graph ? s[0].view_as(s[0]) : s[0].detach(), tx = create_graph ? s[1].view_as(s[1]) : s[1].detach();
      if (!x.requires_grad()) x.set_requires_grad(true);
      if (!tx.requires_grad()) tx.set_requires_grad(true);
      const Tensor ty = at::gelu_backward(tx, x, "tanh");
      const variable_list g = torch::autograd::grad({ty}, {x, tx}, {grads[1]}, /*retain_graph=*/std::nullopt, create_graph);
      dx = dx.defined() ? dx + g[0] : g[0];
      dtx = g[1];
    }
    return {dx, dtx};
  }
};

std::optional<Tensor> gelu(const Tensor& x_) {
  const Route route = find_route();
  Dual x;
  if (!route.ok || !split(x_, route, &x)) return std::nullopt;
  if (attn_dtype(x.p.scalar_type()) < 0 || x.p.numel() == 0) return std::nullopt;
  if (x.t.defined() && (x.t.sizes() != x.p.sizes() || x.t.scalar_type() != x.p.scalar_type() || x.t.device() != x.p.device()))
    return std::nullopt;
  std::optional<BelowTransform> guard(std::in_place, route.jvp);
  Tensor y, ty;
  if (needs_grad({&x.p, &x.t})) {
    try {
      variable_list out = GeluNode::apply(x.p, maybe(x.t));
      y = out[0];
      if (x.t.defined()) ty = out[1];
    } catch (const RejectedError&) {
      return std::nullopt;
    }
  } else {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    PairOut r = gelu_forward(x.p, x.t);
    if (r.status != DMF_ATTN_OK) return std::nullopt;
    y = r.y;
    ty = r.ty;
  }
  guard.reset();
  return put_back(y, ty, route);
}

}  // namespace

PYBIND11_MODULE(_dmf_torch, m) {
  using release = py::call_guard<py::gil_scoped_release>;
  m.def("attn_func", &attn_func, release());
  m.def("attn_qkvpacked", &attn_qkvpacked, release());
  m.def("rms_norm", &rms_norm, release());
  m.def("ln_modulate", &ln_modulate, release());
  m.def("gate_residual", &gate_residual, release());
  m.def("gelu", &gelu, release());
  m.def("set_status_word", [](int64_t device, int64_t ptr) {
    TORCH_CHECK(device >= 0 && device < kMaxDevices, "device index out of range");
    g_status_word[device].store(reinterpret_cast<int32_t*>(ptr), std::memory_order_release);
  });
  m.def("launch_count", [] { return g_launches.load(std::memory_order_relaxed); });
  m.def("add_launches", [](int64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); });
  m.def("set_launch_count", [](int64_t n) { g_launches.store(n, std::memory_order_relaxed); });
}
