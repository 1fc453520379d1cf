// Pieces of the training backward that the recurrence and the fused sub-ops share.
#pragma once
#include "recurrence.h"

namespace lact_torch {

// bf16 operand of a product: [batch][rows][cols] with row / batch strides in elements
struct View {
  const void* p;
  int64_t ld, bs;
  View(const Tensor& t) : p(t.data_ptr()), ld(t.stride(1)), bs(t.stride(0)) {}
  View(const void* p_, int64_t ld_, int64_t bs_) : p(p_), ld(ld_), bs(bs_) {}
};
// tokens [s, ...) of a [B, L, D] bf16 activation
inline View tokens(const Tensor& t, int64_t s) {
  return View(static_cast<const at::BFloat16*>(t.data_ptr()) + s * t.stride(1), t.stride(1), t.stride(0));
}

// c[batch, M, N] (+)= a b^T; a is [M][K] or (mn) [K][M], likewise b
inline lact_bmm_desc product(View a, bool a_mn, View b, bool b_mn, View c, int dtype, bool accumulate, int64_t batch, int64_t M,
                             int64_t N, int64_t K) {
  lact_bmm_desc d;
  std::memset(&d, 0, sizeof(d));
  d.a0 = a.p; d.a0_ld = a.ld; d.a0_bs = a.bs; d.a0_mn = a_mn;
  d.b0 = b.p; d.b0_ld = b.ld; d.b0_bs = b.bs; d.b0_mn = b_mn;
  d.c = const_cast<void*>(c.p); d.c_ld = c.ld; d.c_bs = c.bs;
  d.batch = batch; d.M = M; d.N = N; d.K = K;
  d.c_dtype = dtype; d.accumulate = accumulate;
  return d;
}
inline lact_bmm_desc& plus(lact_bmm_desc& d, View a, bool a_mn, View b, bool b_mn) {
  d.a1 = a.p; d.a1_ld = a.ld; d.a1_bs = a.bs; d.a1_mn = a_mn;
  d.b1 = b.p; d.b1_ld = b.ld; d.b1_bs = b.bs; d.b1_mn = b_mn;
  return d;
}

// Backward of the two token-local stages on one token range.  Scratch planes are allocated once per sweep and token
// count; `w02` / `w1` are the bf16 weights the step computed with.
class TokenBackward {
 public:
  TokenBackward(int64_t B, int64_t D, int64_t H, const Tensor& like, StatusWord status, void* stream)
      : B_(B), D_(D), H_(H), like_(like), status_(std::move(status)), stream_(stream) {}
  // o = w1 (silu(w0 q) * (w2 q)): weight gradients (+)= into dW02 / dW1 (fp32), dq (bf16) written.
  void apply(View w02, View w1, View q, View dO, int64_t n, View dW02, View dW1, bool accumulate, View dq);
  // lr-weighted fast-weight gradient, given the bf16 gradients g02 / g1 of its outputs: weight gradients (+)=, dk, dv
  // (bf16) written, learning-rate gradients (fp32, batch stride glr_bs) written or added.
  void gradient(View w02, View w1, View k, View v, int64_t n, const void* const lr[3], int lr_dtype, int64_t lr_bs, float w_scale,
                View g02, View g1, View dW02, View dW1, bool accumulate, View dk, View dv, float* const glr[3], int64_t glr_bs,
                bool glr_add);

 private:
  void contraction(const lact_bmm_desc* d);  // two products summed over tokens
  View plane(Tensor& t, int64_t n, int64_t width) {
    if (!t.defined() || t.size(1) != n || t.size(2) != width) t = empty({B_, n, width}, at::kBFloat16, like_);
    return View(t);
  }
  int64_t B_, D_, H_;
  Tensor like_;
  StatusWord status_;
  void* stream_;
  Tensor a_, b_, c_, d_, e_, f_, g_, h_;
  Tensor split_, split_count_;  // scratch of split contractions, once one is
};

}  // namespace lact_torch
