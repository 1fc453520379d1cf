// lact_b200::swa_fwd / swa_bwd (sliding-window, causal and block attention) and the sequence-start index.
#include "common.h"

namespace lact_torch {
namespace {

// [b, l, h, d] with heads adjacent within a token and 16-byte aligned token / batch strides (the layout of a slice of a
// fused projection reshaped to heads); anything else is copied
Tensor head_view(const Tensor& t) {
  const int64_t h = t.size(2), d = t.size(3);
  if (t.stride(3) != 1 || t.stride(2) != d || t.stride(1) % 8 || t.stride(0) % 8 || t.stride(1) < h * d ||
      reinterpret_cast<uintptr_t>(t.data_ptr()) % 16)
    return t.contiguous();
  return t;
}

using FwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, int64_t, double, const OptTensor&);
using BwdSig = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, int64_t,
                                   double, const OptTensor&);
const auto& fwd_op() {
  static const auto o = c10::Dispatcher::singleton().findSchemaOrThrow("lact_b200::swa_fwd", "").typed<FwdSig>();
  return o;
}
const auto& bwd_op() {
  static const auto o = c10::Dispatcher::singleton().findSchemaOrThrow("lact_b200::swa_bwd", "").typed<BwdSig>();
  return o;
}

// [o, lse]: the attention output and every row's log-sum-exp (log2 domain, fp32 [b, h, l]) for the backward.
// window > 0: causal, the last `window` keys; 0: causal, all earlier keys; < 0: block attention (not causal: every query
// sees all keys of its batch entry; k and v may then hold another number of tokens than q).
std::vector<Tensor> swa(const Tensor& q_, const Tensor& k_, const Tensor& v_, int64_t window, double scale, const OptTensor& seq) {
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = head_view(q_), k = head_view(k_), v = head_view(v_);
  const int64_t b = q.size(0), l = q.size(1), h = q.size(2), d = q.size(3), lk = k.size(1);
  Tensor o = empty({b, l, h, d}, at::kBFloat16, q), lse = empty({b, h, l}, at::kFloat, q);
  size_t need = 0;
  int64_t words = 0;
  if (lact_swa_fwd_split_bytes(b, l, lk, h, d, window, &need, &words) != LACT_OK) need = 0;  // the call below reports it
  Tensor scratch, counters;
  if (need > 0) {
    scratch = bytes(need, q);
    if (words > 0) counters = at::zeros({words}, q.options().dtype(at::kInt).requires_grad(false));
  }
  void* const room = need > 0 ? ptr(scratch) : nullptr;
  check(lact_swa_fwd_split(ptr(q), ptr(k), ptr(v), ptr(o), b, l, lk, h, d, q.stride(1), q.stride(0), k.stride(1), k.stride(0), v.stride(1),
                     v.stride(0), o.stride(1), o.stride(0), window, static_cast<float>(scale), static_cast<const int32_t*>(ptr(seq)),
                     ptr(lse), words > 0 ? ptr(counters) : room, room, need, status_word(q),
                     stream_of(q)),
        "lact_swa_fwd");
  return {o, lse};
}

// Block attention of q over the keys and values of a cache followed by k, v, where they lie.
Tensor swa_cache(const Tensor& q_, const Tensor& kc_, const Tensor& vc_, const Tensor& k_, const Tensor& v_, double scale) {
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = head_view(q_), kc = head_view(kc_), vc = head_view(vc_), k = head_view(k_), v = head_view(v_);
  const int64_t b = q.size(0), l = q.size(1), h = q.size(2), d = q.size(3), lc = kc.size(1), ln = k.size(1);
  Tensor o = empty({b, l, h, d}, at::kBFloat16, q);
  size_t need = 0;
  int64_t words = 0;
  if (lact_swa_fwd_cache_bytes(b, l, lc, ln, h, d, &need, &words) != LACT_OK) need = 0;  // the call below reports it
  Tensor scratch, counters;
  if (need > 0) {
    scratch = bytes(need, q);
    if (words > 0) counters = at::zeros({words}, q.options().dtype(at::kInt).requires_grad(false));
  }
  void* const room = need > 0 ? ptr(scratch) : nullptr;
  const int64_t strides[12] = {q.stride(1), q.stride(0), kc.stride(1), kc.stride(0), vc.stride(1), vc.stride(0),
                               k.stride(1), k.stride(0), v.stride(1),  v.stride(0),  o.stride(1),  o.stride(0)};
  check(lact_swa_fwd_cache(ptr(q), ptr(kc), ptr(vc), ptr(k), ptr(v), ptr(o), b, l, lc, ln, h, d, strides, static_cast<float>(scale),
                           words > 0 ? ptr(counters) : room, room, need, status_word(q), stream_of(q)),
        "lact_swa_fwd_cache");
  return o;
}

// [dq, dk, dv] (bf16, contiguous): probabilities recomputed from lse
std::vector<Tensor> swa_bwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& o_, const Tensor& lse_,
                            const Tensor& dout_, int64_t window, double scale, const OptTensor& seq) {
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = head_view(q_), k = head_view(k_), v = head_view(v_), o = head_view(o_);
  const Tensor dout = head_view(dout_.to(at::kBFloat16)), lse = lse_.contiguous();
  const int64_t b = q.size(0), l = q.size(1), h = q.size(2), d = q.size(3), lk = k.size(1);
  Tensor dq = empty({b, l, h, d}, at::kBFloat16, q), dk = empty({b, lk, h, d}, at::kBFloat16, q), dv = at::empty_like(dk);
  Tensor delta = empty({b, h, l}, at::kFloat, q);
  check(lact_swa_bwd(ptr(q), ptr(k), ptr(v), ptr(o), ptr(dout), ptr(lse), ptr(dq), ptr(dk), ptr(dv), ptr(delta), b, l, lk, h, d,
                     q.stride(1), q.stride(0), k.stride(1), k.stride(0), v.stride(1), v.stride(0), o.stride(1), o.stride(0),
                     dout.stride(1), dout.stride(0), window, static_cast<float>(scale), static_cast<const int32_t*>(ptr(seq)),
                     status_word(q), stream_of(q)),
        "lact_swa_bwd");
  settle(q);
  return {dq, dk, dv};
}

class SwaFunction : public torch::autograd::Function<SwaFunction> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, int64_t window, double scale,
                               const OptTensor& seq) {
    at::AutoDispatchBelowADInplaceOrView guard;
    variable_list r = fwd_op().call(q, k, v, window, scale, seq);
    ctx->save_for_backward({q, k, v, r[0], r[1], value(seq)});
    ctx->saved_data["window"] = window;
    ctx->saved_data["scale"] = scale;
    ctx->set_materialize_grads(false);
    ctx->mark_non_differentiable({r[1]});
    return r;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto t = ctx->get_saved_variables();
    if (!g[0].defined()) return variable_list(6);
    variable_list r = bwd_op().call(t[0], t[1], t[2], t[3], t[4], g[0], ctx->saved_data["window"].toInt(),
                                    ctx->saved_data["scale"].toDouble(), opt(t[5]));
    r.resize(6);
    return r;
  }
};
std::vector<Tensor> swa_autograd(const Tensor& q, const Tensor& k, const Tensor& v, int64_t window, double scale,
                                 const OptTensor& seq) {
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad()))
    return SwaFunction::apply(q, k, v, window, scale, seq);
  at::AutoDispatchBelowADInplaceOrView guard;
  return fwd_op().call(q, k, v, window, scale, seq);
}

using CacheSig = Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, double);
// (with gradients the keys and values are put together first: the backward reads them as one array)
Tensor swa_cache_autograd(const Tensor& q, const Tensor& kc, const Tensor& vc, const Tensor& k, const Tensor& v, double scale) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("lact_b200::swa_fwd_cache", "").typed<CacheSig>();
  bool grad = false;
  for (const Tensor* t : {&q, &kc, &vc, &k, &v}) grad = grad || t->requires_grad();
  if (at::GradMode::is_enabled() && grad) return fwd_op().call(q, at::cat({kc, k}, 1), at::cat({vc, v}, 1), -1, scale, {})[0];
  at::AutoDispatchBelowADInplaceOrView guard;
  return op.call(q, kc, vc, k, v, scale);
}

// int32 [n_tokens]: first token of the packed sequence every token belongs to
Tensor seq_start(const Tensor& cu_, int64_t n_tokens) {
  const c10::cuda::CUDAGuard guard(cu_.device());
  const Tensor cu = cu_.to(at::kInt).contiguous();
  Tensor out = empty({n_tokens}, at::kInt, cu);
  if (n_tokens > 0)
    check(lact_seq_start(cu.data_ptr<int32_t>(), cu.numel() - 1, n_tokens, out.data_ptr<int32_t>(), stream_of(cu)), "lact_seq_start");
  return out;
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(lact_b200, m) {
  m.def("swa_fwd(Tensor q, Tensor k, Tensor v, int window, float softmax_scale, Tensor? seq_start=None) -> Tensor[]");
  m.def("swa_fwd_cache(Tensor q, Tensor k_cache, Tensor v_cache, Tensor k, Tensor v, float softmax_scale) -> Tensor");
  m.def("swa_bwd(Tensor q, Tensor k, Tensor v, Tensor o, Tensor lse, Tensor dout, int window, float softmax_scale, "
        "Tensor? seq_start=None) -> Tensor[]");
  m.def("seq_start(Tensor cu_seqlens, int n_tokens) -> Tensor");
}
TORCH_LIBRARY_IMPL(lact_b200, CUDA, m) {
  m.impl("swa_fwd", &swa);
  m.impl("swa_fwd_cache", &swa_cache);
  m.impl("swa_bwd", &swa_bwd);
  m.impl("seq_start", &seq_start);
}
TORCH_LIBRARY_IMPL(lact_b200, Autograd, m) {
  m.impl("swa_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("swa_fwd", &swa_autograd);
  m.impl("swa_fwd_cache", &swa_cache_autograd);
}

}  // namespace lact_torch
