// lact_b200::scan_fwd: the chunk recurrence, forward (kernels) and autograd (saves what scan_bwd.cpp reads).
#include <algorithm>

#include "recurrence.h"

namespace lact_torch {
namespace {

// [b, l, 1] or [b, l] per-token scalar -> contiguous, fp32 or bf16
Tensor per_token(const Tensor& t0, int64_t B, int64_t L, const char* name) {
  Tensor t = t0;
  if (t.dim() == 3) {
    TORCH_CHECK_VALUE(t.size(2) == 1, name, " must be [b, l, 1]");
    t = t.select(2, 0);
  }
  TORCH_CHECK_VALUE(t.dim() == 2 && t.size(0) == B && t.size(1) == L, name, " has shape ", t.sizes(), ", expected [", B, ", ", L, "]");
  if (t.scalar_type() != at::kFloat && t.scalar_type() != at::kBFloat16) t = t.to(at::kFloat);
  return t.contiguous();
}

Tensor weight(const Tensor& t0, int64_t B, int64_t R, int64_t C, const char* name) {
  TORCH_CHECK_VALUE(t0.dim() == 3 && t0.size(0) == B && t0.size(1) == R && t0.size(2) == C, name, " has shape ", t0.sizes(),
                    ", expected [", B, ", ", R, ", ", C, "]");
  Tensor t = t0;
  if (t.scalar_type() != at::kFloat && t.scalar_type() != at::kBFloat16) t = t.to(at::kFloat);
  return t.contiguous();
}

void same_dtype(Tensor& a, Tensor& b, Tensor& c) {
  if (a.scalar_type() == b.scalar_type() && b.scalar_type() == c.scalar_type()) return;
  a = a.to(at::kFloat); b = b.to(at::kFloat); c = c.to(at::kFloat);
}

std::vector<Tensor> scan_fwd(const Tensor& w0_, const Tensor& w1_, const Tensor& w2_, const Tensor& q_, const Tensor& k_,
                             const Tensor& v_, const Tensor& lr0_, const Tensor& lr1_, const Tensor& lr2_,
                             const OptTensor& momentum_, const OptTensor& m0, const OptTensor& m1, const OptTensor& m2,
                             at::IntArrayRef steps_, at::IntArrayRef cfg_, double w_scale) {
  const c10::cuda::CUDAGuard guard(k_.device());
  poll_status(k_);
  const Options o(cfg_);
  const Steps st(steps_);
  const bool f32 = q_.scalar_type() == at::kFloat && k_.scalar_type() == at::kFloat && v_.scalar_type() == at::kFloat;
  for (const Tensor* t : {&q_, &k_, &v_}) {
    TORCH_CHECK_TYPE(f32 || t->scalar_type() == at::kBFloat16, "q, k, v must be bfloat16, or all float32 (got ", t->scalar_type(), ")");
    TORCH_CHECK_VALUE(t->dim() == 3, "q, k, v must be [b, l, d]");
  }
  const Tensor mom_ = value(momentum_), state_[3] = {value(m0), value(m1), value(m2)};
  for (const Tensor* t : {&w0_, &w1_, &w2_, &q_, &v_, &lr0_, &lr1_, &lr2_, &mom_, &state_[0], &state_[1], &state_[2]}) {
    if (!t->defined()) continue;
    TORCH_CHECK(t->is_cuda(), "lact_b200 runs on CUDA tensors only (there is no CPU implementation)");
    TORCH_CHECK_VALUE(t->device() == k_.device(), "all tensors must be on the same device");
  }
  const Tensor q = aligned(q_, f32 ? 4 : 8), k = aligned(k_, f32 ? 4 : 8), v = aligned(v_, f32 ? 4 : 8);
  const int64_t B = k.size(0), L = k.size(1), D = k.size(2);
  TORCH_CHECK_VALUE(w0_.dim() == 3, "w0 must be [b, d_h, d]");
  const int64_t H = w0_.size(1);
  TORCH_CHECK_VALUE(q.size(0) == B && q.size(2) == D && v.sizes() == k.sizes(), "q, k, v shapes disagree");
  TORCH_CHECK_VALUE(q.size(1) == L, "q and k must have the same number of tokens");
  Tensor w0 = weight(w0_, B, H, D, "w0"), w1 = weight(w1_, B, D, H, "w1"), w2 = weight(w2_, B, H, D, "w2");
  same_dtype(w0, w1, w2);
  Tensor lr0 = per_token(lr0_, B, L, "lr0"), lr1 = per_token(lr1_, B, L, "lr1"), lr2 = per_token(lr2_, B, L, "lr2");
  same_dtype(lr0, lr1, lr2);
  Tensor mom;
  if (mom_.defined()) mom = per_token(mom_, B, L, "momentum");
  if (mom.defined() && f32) mom = mom.to(at::kFloat);  // (the mean of a bf16 gate is rounded to bf16, as a bf16 model's is)

  lact_scan_config c = base_config(o, B, L, D, H);
  // The reference drivers start from torch.zeros_like(q): tokens no APPLY step covers stay zero.
  Tensor out = empty({B, c.out_len, D}, q.scalar_type(), q);
  for (auto& [s, e] : st.gaps(kApply, c.out_len, true)) out.narrow(1, s, e - s).zero_();
  c.act_dtype = f32 ? LACT_F32 : LACT_BF16;
  c.lr_dtype = dtype_code(lr0);
  c.mom_dtype = mom.defined() ? dtype_code(mom) : LACT_F32;
  c.w_dtype = dtype_code(w0);
  c.use_momentum = mom.defined();
  c.w_scale = static_cast<float>(w_scale);
  c.q_bs = q.stride(0); c.q_ts = q.stride(1);
  c.k_bs = k.stride(0); c.k_ts = k.stride(1);
  c.v_bs = v.stride(0); c.v_ts = v.stride(1);
  c.o_bs = out.stride(0); c.o_ts = out.stride(1);

  lact_scan_io io;
  std::memset(&io, 0, sizeof(io));
  io.w0 = ptr(w0); io.w1 = ptr(w1); io.w2 = ptr(w2);
  io.q = ptr(q); io.k = ptr(k); io.v = ptr(v);
  io.lr0 = ptr(lr0); io.lr1 = ptr(lr1); io.lr2 = ptr(lr2);
  io.momentum = mom.defined() ? ptr(mom) : nullptr;
  io.o = ptr(out);
  Tensor mi[3];
  if (state_[0].defined()) {
    for (int i = 0; i < 3; ++i) {
      TORCH_CHECK_VALUE(state_[i].defined(), "the momentum state has three parts");
      mi[i] = state_[i].to(at::kFloat).contiguous();
      TORCH_CHECK_VALUE(mi[i].numel() == B * D * H, "momentum state: one value per weight");
    }
    io.m0_in = ptr(mi[0]); io.m1_in = ptr(mi[1]); io.m2_in = ptr(mi[2]);
  }
  std::vector<Tensor> res{out};
  auto states = [&](void** a, void** b, void** d) {
    Tensor t[3] = {empty({B, H, D}, at::kFloat, q), empty({B, D, H}, at::kFloat, q), empty({B, H, D}, at::kFloat, q)};
    *a = ptr(t[0]); *b = ptr(t[1]); *d = ptr(t[2]);
    res.insert(res.end(), t, t + 3);
  };
  if (o.return_state) states(&io.w0_out, &io.w1_out, &io.w2_out);
  if (o.return_momentum) states(&io.m0_out, &io.m1_out, &io.m2_out);
  if (o.save) {
    TORCH_CHECK_NOT_IMPLEMENTED(!f32, "fp32 mode is forward only; the training backward runs on bf16 activations");
    const int64_t slots = std::max(st.updates, 1);
    const size_t stride = trace_layout(o, B, L, D, H).first;
    Tensor dump = empty({slots, state_elems(B, D, H)}, at::kFloat, q);
    // with Muon the forward's own Newton-Schulz iterates are kept too (no recomputation in the backward)
    Tensor trace = empty({stride ? slots * static_cast<int64_t>(stride) : 1}, at::kByte, q);
    Tensor shadow = empty({st.updates + 1, 3 * B * D * H}, at::kBFloat16, q);
    io.state_dump = ptr(dump);
    io.ns_trace = stride ? ptr(trace) : nullptr;
    io.shadow_dump = ptr(shadow);
    res.insert(res.end(), {dump, trace, shadow});
  }
  size_t need = 0;
  const auto query = f32 ? lact_scan_f32_workspace_bytes : lact_scan_workspace_bytes;
  check(query(&c, st.n, st.kind.data(), st.start.data(), st.end.data(), &need), "lact_scan_workspace_bytes");
  const Tensor ws = bytes(need, q);
  check((f32 ? lact_scan_f32_fwd : lact_scan_fwd)(&c, &io, st.n, st.kind.data(), st.start.data(), st.end.data(), st.out.data(),
                                                  ptr(ws), static_cast<size_t>(ws.numel()), stream_of(q)),
        "lact_scan_fwd");
  return res;
}

using ScanFwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                       const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const OptTensor&,
                                       const OptTensor&, const OptTensor&, at::IntArrayRef, at::IntArrayRef, double);
using ScanBwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                       const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const Tensor&, const Tensor&,
                                       const Tensor&, const Tensor&, const OptTensor&, const OptTensor&, const OptTensor&,
                                       at::IntArrayRef, at::IntArrayRef, double);
const auto& fwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("lact_b200::scan_fwd", "").typed<ScanFwdSig>();
  return op;
}
const auto& bwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("lact_b200::scan_bwd", "").typed<ScanBwdSig>();
  return op;
}

class ScanFunction : public torch::autograd::Function<ScanFunction> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& w0, const Tensor& w1, const Tensor& w2, const Tensor& q,
                               const Tensor& k, const Tensor& v, const Tensor& lr0, const Tensor& lr1, const Tensor& lr2,
                               const OptTensor& momentum, std::vector<int64_t> steps, std::vector<int64_t> cfg, double w_scale) {
    at::AutoDispatchBelowADInplaceOrView guard;
    cfg[12] = 1;
    const bool state = cfg[13] != 0;
    std::vector<Tensor> r = fwd_op().call(w0, w1, w2, q, k, v, lr0, lr1, lr2, momentum, {}, {}, {}, steps, cfg, w_scale);
    const size_t n = state ? 4 : 1;  // outputs the caller sees; then the saved state
    ctx->save_for_backward({w0, w1, w2, q, k, v, lr0, lr1, lr2, given(momentum) ? *momentum : Tensor(), r[n], r[n + 1], r[n + 2]});
    ctx->saved_data["steps"] = std::move(steps);
    ctx->saved_data["cfg"] = std::move(cfg);
    ctx->saved_data["w_scale"] = w_scale;
    // unused outputs must not arrive in the backward as zero tensors
    ctx->set_materialize_grads(false);
    r.resize(n);
    return r;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    const std::vector<int64_t> steps = ctx->saved_data["steps"].toIntVector(), cfg = ctx->saved_data["cfg"].toIntVector();
    Tensor dO = g[0];
    if (!dO.defined()) dO = at::zeros({t[3].size(0), cfg[10] >= 0 ? cfg[10] : t[4].size(1), t[3].size(2)}, t[3].options());
    OptTensor gw[3];
    for (int i = 0; i < 3; ++i)
      if (g.size() > 1 && g[1 + i].defined()) gw[i] = g[1 + i];
    std::vector<Tensor> d = bwd_op().call(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], opt(t[9]), t[10], t[11], t[12],
                                          dO, gw[0], gw[1], gw[2], steps, cfg, ctx->saved_data["w_scale"].toDouble());
    variable_list out(d.begin(), d.begin() + 9);
    out.push_back(t[9].defined() ? d[9] : Tensor());
    out.resize(13);
    return out;
  }
};

std::vector<Tensor> scan_autograd(const Tensor& w0, const Tensor& w1, const Tensor& w2, const Tensor& q, const Tensor& k,
                                  const Tensor& v, const Tensor& lr0, const Tensor& lr1, const Tensor& lr2,
                                  const OptTensor& momentum, const OptTensor& m0, const OptTensor& m1, const OptTensor& m2,
                                  at::IntArrayRef steps, at::IntArrayRef cfg, double w_scale) {
  bool grad = false;
  if (at::GradMode::is_enabled()) {
    for (const Tensor* t : {&w0, &w1, &w2, &q, &k, &v, &lr0, &lr1, &lr2}) grad = grad || t->requires_grad();
    grad = grad || (given(momentum) && momentum->requires_grad());
  }
  if (!grad) {
    at::AutoDispatchBelowADInplaceOrView guard;
    return fwd_op().call(w0, w1, w2, q, k, v, lr0, lr1, lr2, momentum, m0, m1, m2, steps, cfg, w_scale);
  }
  const Options o(cfg);
  TORCH_CHECK_NOT_IMPLEMENTED(!given(m0) && !o.return_momentum,
                              "gradients through a momentum state passed in / returned are not implemented");
  TORCH_CHECK_NOT_IMPLEMENTED(q.scalar_type() != at::kFloat,
                              "fp32 mode is forward only; the training backward runs on bf16 activations");
  TORCH_CHECK_NOT_IMPLEMENTED(!(o.prenorm && o.overwrite), "no reference recurrence combines pre-norm with the bidirectional overwrite");
  return ScanFunction::apply(w0, w1, w2, q, k, v, lr0, lr1, lr2, momentum, steps.vec(), cfg.vec(), w_scale);
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(lact_b200, m) {
  m.def("scan_fwd(Tensor w0, Tensor w1, Tensor w2, Tensor q, Tensor k, Tensor v, Tensor lr0, Tensor lr1, Tensor lr2, "
        "Tensor? momentum, Tensor? m0, Tensor? m1, Tensor? m2, int[] steps, int[] cfg, float w_scale) -> Tensor[]");
}
TORCH_LIBRARY_IMPL(lact_b200, CUDA, m) { m.impl("scan_fwd", &scan_fwd); }
TORCH_LIBRARY_IMPL(lact_b200, Autograd, m) { m.impl("scan_fwd", &scan_autograd); }

}  // namespace lact_torch
