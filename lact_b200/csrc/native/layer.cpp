// The layer's row-wise passes (q / k / v prologue, learning rates, output epilogue) and attention: kernels and autograd.
#include "common.h"

namespace lact_torch {
namespace {

template <class Sig>
auto op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}
bool wants_grad(const Tensor& t) { return t.defined() && t.requires_grad(); }

// [b, s, n] bf16 rows for the row passes; `flat`: rows of all batch entries evenly spaced (one row stride)
Tensor rows(const Tensor& t, const char* name, bool flat = false) {
  TORCH_CHECK(t.dim() == 3 && t.scalar_type() == at::kBFloat16, name, ": expected a [b, s, n_heads * d] bf16 tensor");
  Tensor r = aligned(t);
  if (flat && r.stride(0) != r.size(1) * r.stride(1)) r = r.contiguous();
  return r;
}

// ---------------------------------------------------------------- qkv_prologue
using QkvSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, int64_t, bool, bool, const OptTensor&,
                                   const OptTensor&, int64_t, int64_t, const OptTensor&);
using QkvBwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const OptTensor&,
                                      const OptTensor&, int64_t, bool, bool, const OptTensor&, const OptTensor&, int64_t, int64_t,
                                      const OptTensor&);
const auto& qkv_op() { static const auto o = op<QkvSig>("lact_b200::qkv_prologue"); return o; }
const auto& qkv_bwd_op() { static const auto o = op<QkvBwdSig>("lact_b200::qkv_prologue_bwd"); return o; }

std::vector<Tensor> qkv(const Tensor& xq_, const Tensor& xk_, const Tensor& xv_, int64_t n_h, bool silu, bool v_silu,
                        const OptTensor& cos, const OptTensor& sin, int64_t hd, int64_t offset, const OptTensor& seq) {
  const c10::cuda::CUDAGuard guard(xq_.device());
  const Tensor x[3] = {rows(xq_, "xq"), rows(xk_, "xk"), rows(xv_, "xv")};
  const int64_t b = x[0].size(0), s = x[0].size(1), d = x[0].size(2) / n_h;
  std::vector<Tensor> r(3);
  for (Tensor& t : r) t = empty({b * n_h, s, d}, at::kBFloat16, x[0]);
  if (!given(cos))
    check(lact_qkv_prologue(ptr(x[0]), ptr(x[1]), ptr(x[2]), x[0].stride(1), x[1].stride(1), x[2].stride(1), x[0].stride(0),
                            x[1].stride(0), x[2].stride(0), ptr(r[0]), ptr(r[1]), ptr(r[2]), b, s, n_h, d, silu, v_silu,
                            stream_of(x[0])),
          "lact_qkv_prologue");
  else
    check(lact_qkv_prologue_rope(ptr(x[0]), ptr(x[1]), ptr(x[2]), x[0].stride(1), x[1].stride(1), x[2].stride(1), x[0].stride(0),
                                 x[1].stride(0), x[2].stride(0), ptr(r[0]), ptr(r[1]), ptr(r[2]), b, s, n_h, d, silu, v_silu,
                                 ptr(cos), ptr(sin), hd, cos->size(0), offset, static_cast<const int32_t*>(ptr(seq)),
                                 stream_of(x[0])),
          "lact_qkv_prologue_rope");
  return r;
}

// on the saved projections: rotation transposed, l2 norm and SiLU differentiated in one pass per row
std::vector<Tensor> qkv_bwd(const Tensor& xq_, const Tensor& xk_, const Tensor& xv_, const OptTensor& dq, const OptTensor& dk,
                            const OptTensor& dv, int64_t n_h, bool silu, bool v_silu, const OptTensor& cos, const OptTensor& sin,
                            int64_t hd, int64_t offset, const OptTensor& seq) {
  const c10::cuda::CUDAGuard guard(xq_.device());
  const Tensor x[3] = {rows(xq_, "xq"), rows(xk_, "xk"), rows(xv_, "xv")};
  const int64_t b = x[0].size(0), s = x[0].size(1), nd = x[0].size(2), d = nd / n_h;
  const OptTensor* g[3] = {&dq, &dk, &dv};
  Tensor z[3];
  std::vector<Tensor> r(3);
  for (int i = 0; i < 3; ++i) {
    if (given(*g[i])) z[i] = (*g[i])->to(at::kBFloat16).contiguous();
    r[i] = empty({b, s, nd}, at::kBFloat16, x[0]);
  }
  auto p = [](const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; };
  check(lact_qkv_prologue_bwd(ptr(x[0]), ptr(x[1]), ptr(x[2]), x[0].stride(1), x[1].stride(1), x[2].stride(1), x[0].stride(0),
                              x[1].stride(0), x[2].stride(0), p(z[0]), p(z[1]), p(z[2]), ptr(r[0]), ptr(r[1]), ptr(r[2]), b, s, n_h,
                              d, silu, v_silu, ptr(cos), ptr(sin), given(cos) ? hd : 0, given(cos) ? cos->size(0) : 0, offset,
                              static_cast<const int32_t*>(ptr(seq)), stream_of(x[0])),
        "lact_qkv_prologue_bwd");
  return r;
}

class QkvFunction : public torch::autograd::Function<QkvFunction> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& xq, const Tensor& xk, const Tensor& xv, int64_t n_h, bool silu,
                               bool v_silu, const OptTensor& cos, const OptTensor& sin, int64_t hd, int64_t offset, const OptTensor& seq) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({xq, xk, xv, value(cos), value(sin), value(seq)});
    ctx->saved_data["cfg"] = std::vector<int64_t>{n_h, silu, v_silu, hd, offset};
    ctx->set_materialize_grads(false);
    return qkv_op().call(xq, xk, xv, n_h, silu, v_silu, cos, sin, hd, offset, seq);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    const auto c = ctx->saved_data["cfg"].toIntVector();
    variable_list r = qkv_bwd_op().call(t[0], t[1], t[2], opt(g[0]), opt(g[1]), opt(g[2]), c[0], c[1] != 0, c[2] != 0, opt(t[3]),
                                        opt(t[4]), c[3], c[4], opt(t[5]));
    r.resize(11);
    return r;
  }
};
std::vector<Tensor> qkv_autograd(const Tensor& xq, const Tensor& xk, const Tensor& xv, int64_t n_h, bool silu, bool v_silu,
                                 const OptTensor& cos, const OptTensor& sin, int64_t hd, int64_t offset, const OptTensor& seq) {
  if (at::GradMode::is_enabled() && (wants_grad(xq) || wants_grad(xk) || wants_grad(xv)))
    return QkvFunction::apply(xq, xk, xv, n_h, silu, v_silu, cos, sin, hd, offset, seq);
  at::AutoDispatchBelowADInplaceOrView guard;
  return qkv_op().call(xq, xk, xv, n_h, silu, v_silu, cos, sin, hd, offset, seq);
}

// ---------------------------------------------------------------- lr_prologue
using LrSig = std::vector<Tensor>(const Tensor&, const OptTensor&, int64_t, double);
using LrBwdSig = std::vector<Tensor>(const Tensor&, const OptTensor&, const OptTensor&, const OptTensor&, const OptTensor&,
                                     const OptTensor&, int64_t, double);
const auto& lr_op() { static const auto o = op<LrSig>("lact_b200::lr_prologue"); return o; }
const auto& lr_bwd_op() { static const auto o = op<LrBwdSig>("lact_b200::lr_prologue_bwd"); return o; }

Tensor flat_rows(const Tensor& t) { return t.stride(2) != 1 || t.stride(0) != t.size(1) * t.stride(1) ? t.contiguous() : t; }

std::vector<Tensor> lr(const Tensor& proj_, const OptTensor& logits_, int64_t n_h, double base_inv) {
  const c10::cuda::CUDAGuard guard(proj_.device());
  const Tensor proj = flat_rows(proj_);
  const int64_t b = proj.size(0), s = proj.size(1);
  Tensor lg;
  if (given(logits_)) lg = flat_rows(*logits_);
  std::vector<Tensor> r(lg.defined() ? 4 : 3);
  for (Tensor& t : r) t = empty({b * n_h, s, 1}, at::kFloat, proj);
  check(lact_lr_prologue(ptr(proj), dtype_code(proj), proj.stride(1), static_cast<float>(base_inv), lg.defined() ? ptr(lg) : nullptr,
                         lg.defined() ? dtype_code(lg) : LACT_F32, lg.defined() ? lg.stride(1) : 0, ptr(r[0]), ptr(r[1]), ptr(r[2]),
                         lg.defined() ? ptr(r[3]) : nullptr, b, s, n_h, stream_of(proj)),
        "lact_lr_prologue");
  return r;
}

std::vector<Tensor> lr_bwd(const Tensor& proj_, const OptTensor& logits_, const OptTensor& g0, const OptTensor& g1,
                           const OptTensor& g2, const OptTensor& gm, int64_t n_h, double base_inv) {
  const c10::cuda::CUDAGuard guard(proj_.device());
  const Tensor proj = flat_rows(proj_);
  const int64_t b = proj.size(0), s = proj.size(1);
  Tensor lg, g[4];
  if (given(logits_)) lg = flat_rows(*logits_);
  const OptTensor* gs[4] = {&g0, &g1, &g2, &gm};
  const void* gp[4];
  for (int i = 0; i < 4; ++i) {
    if (given(*gs[i])) g[i] = (*gs[i])->to(at::kFloat).contiguous();
    gp[i] = g[i].defined() ? ptr(g[i]) : nullptr;
  }
  std::vector<Tensor> r{empty({b, s, 3 * n_h}, proj.scalar_type(), proj)};
  if (lg.defined()) r.push_back(empty({b, s, n_h}, lg.scalar_type(), proj));
  check(lact_lr_prologue_bwd(ptr(proj), dtype_code(proj), proj.stride(1), static_cast<float>(base_inv),
                             lg.defined() ? ptr(lg) : nullptr, lg.defined() ? dtype_code(lg) : LACT_F32,
                             lg.defined() ? lg.stride(1) : 0, gp[0], gp[1], gp[2], gp[3], ptr(r[0]),
                             lg.defined() ? ptr(r[1]) : nullptr, b, s, n_h, stream_of(proj)),
        "lact_lr_prologue_bwd");
  return r;
}

class LrFunction : public torch::autograd::Function<LrFunction> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& proj, const OptTensor& logits, int64_t n_h, double base_inv) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({proj, value(logits)});
    ctx->saved_data["n_h"] = n_h;
    ctx->saved_data["base"] = base_inv;
    ctx->set_materialize_grads(false);
    return lr_op().call(proj, logits, n_h, base_inv);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    g.resize(4);
    const variable_list r = lr_bwd_op().call(t[0], opt(t[1]), opt(g[0]), opt(g[1]), opt(g[2]), opt(g[3]),
                                             ctx->saved_data["n_h"].toInt(), ctx->saved_data["base"].toDouble());
    return {r[0], r.size() > 1 ? r[1] : Tensor(), Tensor(), Tensor()};
  }
};
std::vector<Tensor> lr_autograd(const Tensor& proj, const OptTensor& logits, int64_t n_h, double base_inv) {
  if (at::GradMode::is_enabled() && (wants_grad(proj) || (given(logits) && wants_grad(*logits))))
    return LrFunction::apply(proj, logits, n_h, base_inv);
  at::AutoDispatchBelowADInplaceOrView guard;
  return lr_op().call(proj, logits, n_h, base_inv);
}

// ---------------------------------------------------------------- out_epilogue
using OutSig = Tensor(const Tensor&, const Tensor&, const OptTensor&, const OptTensor&, int64_t, double);
using OutBwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const OptTensor&, const Tensor&, int64_t, double);
const auto& out_op() { static const auto o = op<OutSig>("lact_b200::out_epilogue"); return o; }
const auto& out_bwd_op() { static const auto o = op<OutBwdSig>("lact_b200::out_epilogue_bwd"); return o; }

Tensor out_epi(const Tensor& x_, const Tensor& w_, const OptTensor& gate_, const OptTensor& res_, int64_t n_h, double eps) {
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = x_.contiguous(), w = w_.to(at::kFloat).contiguous();
  const int64_t s = x.size(1), d = x.size(2), b = x.size(0) / n_h;
  Tensor gate, res, out = empty({b, s, n_h * d}, at::kBFloat16, x);
  if (given(gate_)) gate = rows(*gate_, "scale_proj", true);
  if (given(res_)) res = rows(*res_, "o", true);
  check(lact_out_epilogue(ptr(x), ptr(w), gate.defined() ? ptr(gate) : nullptr, gate.defined() ? gate.stride(1) : 0,
                          res.defined() ? ptr(res) : nullptr, res.defined() ? res.stride(1) : 0, ptr(out), out.stride(1), b, s, n_h,
                          d, static_cast<float>(eps), stream_of(x)),
        "lact_out_epilogue");
  return out;
}

// dx, dw (fp32 [d]), dgate (if there is a gate)
std::vector<Tensor> out_epi_bwd(const Tensor& x_, const Tensor& w_, const OptTensor& gate_, const Tensor& dout, int64_t n_h,
                                double eps) {
  const c10::cuda::CUDAGuard guard(x_.device());
  const Tensor x = x_.contiguous(), w = w_.to(at::kFloat).contiguous();
  const int64_t s = x.size(1), d = x.size(2), b = x.size(0) / n_h;
  const Tensor dy = rows(dout.to(at::kBFloat16), "grad", true);
  Tensor gate, dx = at::empty_like(x), dgate, dw = empty({d}, at::kFloat, x);
  if (given(gate_)) {
    gate = rows(*gate_, "scale_proj", true);
    dgate = empty({b, s, n_h * d}, at::kBFloat16, x);
  }
  Tensor part = empty({lact_out_epilogue_bwd_blocks(), d}, at::kFloat, x);
  void* const stream = stream_of(x);
  check(lact_out_epilogue_bwd(ptr(x), ptr(w), gate.defined() ? ptr(gate) : nullptr, gate.defined() ? gate.stride(1) : 0, ptr(dy),
                              dy.stride(1), ptr(dx), gate.defined() ? ptr(dgate) : nullptr, ptr(part), b, s, n_h, d,
                              static_cast<float>(eps), stream),
        "lact_out_epilogue_bwd");
  check(lact_column_sums(part.data_ptr<float>(), dw.data_ptr<float>(), part.size(0), d, stream), "lact_column_sums");
  std::vector<Tensor> r{dx, dw};
  if (gate.defined()) r.push_back(dgate);
  return r;
}

class OutFunction : public torch::autograd::Function<OutFunction> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& gate, const OptTensor& res, int64_t n_h,
                        double eps) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({x, w, value(gate)});
    ctx->saved_data["n_h"] = n_h;
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["res"] = given(res);
    return out_op().call(x, w, gate, res, n_h, eps);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    const auto r = out_bwd_op().call(t[0], t[1], opt(t[2]), g[0], ctx->saved_data["n_h"].toInt(), ctx->saved_data["eps"].toDouble());
    return {r[0], r[1].to(t[1].scalar_type()), r.size() > 2 ? r[2] : Tensor(), ctx->saved_data["res"].toBool() ? g[0] : Tensor(),
            Tensor(), Tensor()};
  }
};
Tensor out_autograd(const Tensor& x, const Tensor& w, const OptTensor& gate, const OptTensor& res, int64_t n_h, double eps) {
  if (at::GradMode::is_enabled() && (wants_grad(x) || wants_grad(w) || wants_grad(value(gate)) || wants_grad(value(res))))
    return OutFunction::apply(x, w, gate, res, n_h, eps);
  at::AutoDispatchBelowADInplaceOrView guard;
  return out_op().call(x, w, gate, res, n_h, eps);
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(lact_b200, m) {
  m.def("qkv_prologue(Tensor xq, Tensor xk, Tensor xv, int n_heads, bool silu, bool v_silu, Tensor? cos, Tensor? sin, "
        "int rope_head_dim, int offset, Tensor? seq_start) -> Tensor[]");
  m.def("qkv_prologue_bwd(Tensor xq, Tensor xk, Tensor xv, Tensor? dq, Tensor? dk, Tensor? dv, int n_heads, bool silu, bool v_silu, "
        "Tensor? cos, Tensor? sin, int rope_head_dim, int offset, Tensor? seq_start) -> Tensor[]");
  m.def("lr_prologue(Tensor proj, Tensor? logits, int n_heads, float base_lr_inv) -> Tensor[]");
  m.def("lr_prologue_bwd(Tensor proj, Tensor? logits, Tensor? g0, Tensor? g1, Tensor? g2, Tensor? gm, int n_heads, "
        "float base_lr_inv) -> Tensor[]");
  m.def("out_epilogue(Tensor fw_x, Tensor norm_weight, Tensor? scale_proj, Tensor? o, int n_heads, float eps) -> Tensor");
  m.def("out_epilogue_bwd(Tensor fw_x, Tensor norm_weight, Tensor? scale_proj, Tensor dout, int n_heads, float eps) -> Tensor[]");
}
TORCH_LIBRARY_IMPL(lact_b200, CUDA, m) {
  m.impl("qkv_prologue", &qkv);
  m.impl("qkv_prologue_bwd", &qkv_bwd);
  m.impl("lr_prologue", &lr);
  m.impl("lr_prologue_bwd", &lr_bwd);
  m.impl("out_epilogue", &out_epi);
  m.impl("out_epilogue_bwd", &out_epi_bwd);
}
TORCH_LIBRARY_IMPL(lact_b200, Autograd, m) {
  m.impl("qkv_prologue_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("lr_prologue_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("out_epilogue_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("qkv_prologue", &qkv_autograd);
  m.impl("lr_prologue", &lr_autograd);
  m.impl("out_epilogue", &out_autograd);
}

}  // namespace lact_torch
