// The fused sub-ops the reference wraps in autograd Functions (FusedSwiGLUFFNFwd, FusedLactSwiGLUFFNBwd, L2NormAddFunction):
// kernels and autograd formulas.
#include "scan_bwd.h"

namespace lact_torch {
namespace {

template <class Sig>
auto op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}

bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// ---------------------------------------------------------------- swiglu_ffn
using FfnSig = Tensor(const Tensor&, const Tensor&, const Tensor&);
using FfnBwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&);
const auto& ffn_op() { static const auto o = op<FfnSig>("lact_b200::swiglu_ffn_fwd"); return o; }
const auto& ffn_bwd_op() { static const auto o = op<FfnBwdSig>("lact_b200::swiglu_ffn_bwd"); return o; }

Tensor ffn(const Tensor& w02_, const Tensor& w1_, const Tensor& x_) {
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor w02 = w02_.contiguous(), w1 = w1_.contiguous(), x = x_.contiguous();
  const int64_t B = x.size(0), N = x.size(1), D = x.size(2), H = w02.size(1) / 2;
  size_t need = 0;
  if (lact_swiglu_ffn_hidden_bytes(B, N, D, H, &need) != LACT_OK) need = 0;  // the call below reports it
  Tensor out = empty({B, N, D}, at::kBFloat16, x), hidden;
  if (need > 0) hidden = bytes(need, x);
  check(lact_swiglu_ffn_apply(ptr(w02), ptr(w1), ptr(x), ptr(out), need > 0 ? ptr(hidden) : nullptr, B, N, D, H, status_word(x),
                              stream_of(x)),
        "lact_swiglu_ffn_fwd");
  return out;
}

// (grad_W0_W2, grad_W1, grad_X), bf16: lact_swiglu_ffn.py:46-76 (pre-activations recomputed)
std::vector<Tensor> ffn_bwd(const Tensor& w02_, const Tensor& w1_, const Tensor& x_, const Tensor& g_) {
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor w02 = w02_.contiguous(), w1 = w1_.contiguous(), x = aligned(x_), g = aligned(g_.to(at::kBFloat16));
  const int64_t B = x.size(0), N = x.size(1), D = x.size(2), H = w02.size(1) / 2;
  Tensor dw02 = empty(w02.sizes(), at::kFloat, x), dw1 = empty(w1.sizes(), at::kFloat, x), dx = empty({B, N, D}, at::kBFloat16, x);
  TokenBackward tok(B, D, H, x, status_word(x), stream_of(x));
  tok.apply(View(w02), View(w1), View(x), View(g), N, View(dw02), View(dw1), false, View(dx));
  settle(x);
  return {dw02.to(at::kBFloat16), dw1.to(at::kBFloat16), dx};
}

class FfnFunction : public torch::autograd::Function<FfnFunction> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& w02, const Tensor& w1, const Tensor& x) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({w02, w1, x});
    return ffn_op().call(w02, w1, x);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    return ffn_bwd_op().call(t[0], t[1], t[2], g[0]);
  }
};
Tensor ffn_autograd(const Tensor& w02, const Tensor& w1, const Tensor& x) {
  if (wants_grad({&w02, &w1, &x})) return FfnFunction::apply(w02, w1, x);
  at::AutoDispatchBelowADInplaceOrView guard;
  return ffn_op().call(w02, w1, x);
}

// ---------------------------------------------------------------- fw_grads
using GradsSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                     const Tensor&);
using GradsBwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                        const Tensor&, const Tensor&, const Tensor&);
const auto& grads_op() { static const auto o = op<GradsSig>("lact_b200::fw_grads_fwd"); return o; }
const auto& grads_bwd_op() { static const auto o = op<GradsBwdSig>("lact_b200::fw_grads_bwd"); return o; }

std::vector<Tensor> grads(const Tensor& w02, const Tensor& w1, const Tensor& k, const Tensor& v, const Tensor& lr0,
                          const Tensor& lr1, const Tensor& lr2) {
  const c10::cuda::CUDAGuard guard(k.device());
  poll_status(k);
  const int64_t B = k.size(0), N = k.size(1), D = k.size(2), H = w02.size(1) / 2;
  Tensor dw02 = empty({B, 2 * H, D}, at::kBFloat16, k), dw1 = empty({B, D, H}, at::kBFloat16, k);
  size_t need = 0;
  check(lact_fw_grad_workspace_bytes(B, N, D, H, &need), "lact_fw_grad_workspace_bytes");
  const Tensor ws = bytes(need, k);
  check(lact_fw_grad(ptr(w02), ptr(w1), ptr(k), ptr(v), ptr(lr0), ptr(lr1), ptr(lr2), dtype_code(lr0), ptr(dw02), ptr(dw1), B, N, D,
                     H, ptr(ws), ws.numel(), stream_of(k)),
        "lact_fw_grad");
  return {dw02, dw1};
}

// Gradients of (W0_W2, W1, K, V, lr0, lr1, lr2) given those of (DW0_DW2, DW1): lact_fw_grad.py:61-156 (bf16 for weights and
// activations, fp32 row sums for the learning rates)
std::vector<Tensor> grads_bwd(const Tensor& w02, const Tensor& w1, const Tensor& k_, const Tensor& v_, const Tensor& lr0,
                              const Tensor& lr1, const Tensor& lr2, const Tensor& g02_, const Tensor& g1_) {
  const c10::cuda::CUDAGuard guard(k_.device());
  const auto BF = at::kBFloat16;
  const Tensor k = aligned(k_), v = aligned(v_), g02 = g02_.to(BF).contiguous(), g1 = g1_.to(BF).contiguous();
  const int64_t B = k.size(0), N = k.size(1), D = k.size(2), H = w02.size(1) / 2;
  Tensor dw02 = empty(w02.sizes(), at::kFloat, k), dw1 = empty(w1.sizes(), at::kFloat, k);
  Tensor dk = empty({B, N, D}, BF, k), dv = empty({B, N, D}, BF, k), glr[3];
  for (Tensor& t : glr) t = empty({B, N}, at::kFloat, k);
  const Tensor l[3] = {lr0.contiguous(), lr1.contiguous(), lr2.contiguous()};
  const void* lp[3] = {ptr(l[0]), ptr(l[1]), ptr(l[2])};
  float* gp[3] = {glr[0].data_ptr<float>(), glr[1].data_ptr<float>(), glr[2].data_ptr<float>()};
  TokenBackward tok(B, D, H, k, status_word(k), stream_of(k));
  tok.gradient(View(w02), View(w1), View(k), View(v), N, lp, dtype_code(lr0), N, 1.0f, View(g02), View(g1), View(dw02), View(dw1),
               false, View(dk), View(dv), gp, N, false);
  settle(k);
  return {dw02.to(BF), dw1.to(BF), dk, dv, glr[0].to(lr0.scalar_type()), glr[1].to(lr1.scalar_type()), glr[2].to(lr2.scalar_type())};
}

class GradsFunction : public torch::autograd::Function<GradsFunction> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& w02, const Tensor& w1, const Tensor& k, const Tensor& v,
                               const Tensor& lr0, const Tensor& lr1, const Tensor& lr2) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({w02, w1, k, v, lr0, lr1, lr2});
    ctx->set_materialize_grads(false);
    return grads_op().call(w02, w1, k, v, lr0, lr1, lr2);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    const Tensor g02 = g[0].defined() ? g[0] : at::zeros_like(t[0]), g1 = g[1].defined() ? g[1] : at::zeros_like(t[1]);
    return grads_bwd_op().call(t[0], t[1], t[2], t[3], t[4], t[5], t[6], g02, g1);
  }
};
std::vector<Tensor> grads_autograd(const Tensor& w02, const Tensor& w1, const Tensor& k, const Tensor& v, const Tensor& lr0,
                                   const Tensor& lr1, const Tensor& lr2) {
  if (wants_grad({&w02, &w1, &k, &v, &lr0, &lr1, &lr2})) return GradsFunction::apply(w02, w1, k, v, lr0, lr1, lr2);
  at::AutoDispatchBelowADInplaceOrView guard;
  return grads_op().call(w02, w1, k, v, lr0, lr1, lr2);
}

// ---------------------------------------------------------------- l2_norm_add
using L2Sig = Tensor(const Tensor&, const Tensor&, const Tensor&, double, bool);
using L2BwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, double);
const auto& l2_op() { static const auto o = op<L2Sig>("lact_b200::l2_norm_add_fwd"); return o; }
const auto& l2_bwd_op() { static const auto o = op<L2BwdSig>("lact_b200::l2_norm_add_bwd"); return o; }

Tensor l2(const Tensor& x_, const Tensor& xa_, const Tensor& scale, double eps, bool out_bf16) {
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = x_.contiguous(), xa = xa_.contiguous();
  const int64_t B = x.size(0), T = x.size(1), D = x.size(2);
  const Tensor sc = scale.reshape({B, T}).to(at::kFloat).contiguous();
  Tensor y = empty({B, T, D}, out_bf16 ? at::kBFloat16 : at::kFloat, x);
  check(lact_l2_norm_add(ptr(x), dtype_code(x), ptr(xa), dtype_code(xa), ptr(sc), ptr(y), dtype_code(y), B, T, D,
                         static_cast<float>(eps), stream_of(x)),
        "lact_l2_norm_add");
  return y;
}

// (dx, dx_add, dtgt_scale) of y = (x + x_add) * rsqrt(sum (x + x_add)^2 + eps) * tgt_scale
// (l2norm_triton_kernels.py:97-172, 409-416); the row is recomputed from the inputs
std::vector<Tensor> l2_bwd(const Tensor& x_, const Tensor& xa_, const Tensor& scale, const Tensor& dy_, double eps) {
  const c10::cuda::CUDAGuard guard(x_.device());
  TORCH_CHECK_NOT_IMPLEMENTED(std::abs(eps - 1e-5) <= 1e-12,
                              "the backward of l2_norm_add_fused is built for eps = 1e-5 (the value every caller uses)");
  const int64_t B = x_.size(0), T = x_.size(1), D = x_.size(2);
  const auto F = at::kFloat;
  const Tensor x = x_.to(F).contiguous(), xa = xa_.contiguous(), dy = dy_.to(F).contiguous();
  const Tensor sc = scale.reshape({B, T}).to(F).contiguous();
  Tensor dsc = at::zeros({B, T}, sc.options()), dw = empty({B, T, D}, F, x);
  check(lact_renorm_bwd(ptr(x), ptr(xa), dtype_code(xa), ptr(sc), ptr(dy), ptr(dw), nullptr, ptr(dsc), B * T, D,
                        LACT_RENORM_EPS_INSIDE, stream_of(x)),
        "lact_renorm_bwd");
  // (two distinct tensors even where both inputs have dw's dtype: an operator's outputs may not alias one another)
  Tensor dxa = xa_.scalar_type() != F ? dw.to(xa_.scalar_type()) : dw.clone();
  return {dw.to(x_.scalar_type()), dxa, dsc.reshape(scale.sizes()).to(scale.scalar_type())};
}

class L2Function : public torch::autograd::Function<L2Function> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& xa, const Tensor& scale, double eps, bool out_bf16) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({x, xa, scale});
    ctx->saved_data["eps"] = eps;
    return l2_op().call(x, xa, scale, eps, out_bf16);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    variable_list d = l2_bwd_op().call(t[0], t[1], t[2], g[0], ctx->saved_data["eps"].toDouble());
    d.resize(5);
    return d;
  }
};
Tensor l2_autograd(const Tensor& x, const Tensor& xa, const Tensor& scale, double eps, bool out_bf16) {
  if (wants_grad({&x, &xa, &scale})) return L2Function::apply(x, xa, scale, eps, out_bf16);
  at::AutoDispatchBelowADInplaceOrView guard;
  return l2_op().call(x, xa, scale, eps, out_bf16);
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(lact_b200, m) {
  m.def("swiglu_ffn_fwd(Tensor W0_W2, Tensor W1, Tensor X) -> Tensor");
  m.def("swiglu_ffn_bwd(Tensor W0_W2, Tensor W1, Tensor X, Tensor grad_out) -> Tensor[]");
  m.def("fw_grads_fwd(Tensor W0_W2, Tensor W1, Tensor K, Tensor V, Tensor lr0, Tensor lr1, Tensor lr2) -> Tensor[]");
  m.def("fw_grads_bwd(Tensor W0_W2, Tensor W1, Tensor K, Tensor V, Tensor lr0, Tensor lr1, Tensor lr2, Tensor g02, Tensor g1) "
        "-> Tensor[]");
  m.def("l2_norm_add_fwd(Tensor x, Tensor x_add, Tensor tgt_scale, float eps, bool out_bf16) -> Tensor");
  m.def("l2_norm_add_bwd(Tensor x, Tensor x_add, Tensor tgt_scale, Tensor dy, float eps) -> Tensor[]");
}
TORCH_LIBRARY_IMPL(lact_b200, CUDA, m) {
  m.impl("swiglu_ffn_fwd", &ffn);
  m.impl("swiglu_ffn_bwd", &ffn_bwd);
  m.impl("fw_grads_fwd", &grads);
  m.impl("fw_grads_bwd", &grads_bwd);
  m.impl("l2_norm_add_fwd", &l2);
  m.impl("l2_norm_add_bwd", &l2_bwd);
}
TORCH_LIBRARY_IMPL(lact_b200, Autograd, m) {
  m.impl("swiglu_ffn_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("fw_grads_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("l2_norm_add_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("swiglu_ffn_fwd", &ffn_autograd);
  m.impl("fw_grads_fwd", &grads_autograd);
  m.impl("l2_norm_add_fwd", &l2_autograd);
}

}  // namespace lact_torch
