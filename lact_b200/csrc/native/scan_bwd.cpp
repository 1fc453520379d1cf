// lact_b200::scan_bwd: training backward of the chunk recurrence, chunk by chunk in reverse.
//
// The structure follows the reference's hand-written backward of its two fused autograd Functions
// (lact_llm/lact_model/lact_triton_kernels/lact_swiglu_ffn.py:46-76 and lact_fw_grad.py:61-156) and autograd through the
// eager momentum / renormalisation lines (ttt_operation.py:170-200).  Pre-activations are recomputed in bf16; activation
// gradients are bf16, weight, learning-rate and momentum gradients fp32 sums.  Weights, gradients and Newton-Schulz
// iterates of every update come from the state the training forward kept.
//
// Driven from Python the sweep takes about 35 us of host time per launch, 2.2 ms for a program of one update whose kernels take
// 1.1 ms.
#include <algorithm>

#include "scan_bwd.h"

namespace lact_torch {

void TokenBackward::contraction(const lact_bmm_desc* d) {
  size_t need = 0;
  int64_t words = 0;
  check(lact_bmm_group_split_bytes(d, 2, &need, &words), "lact_bmm_group_split_bytes");
  if (need > 0 && (!split_count_.defined() || split_count_.numel() < words))
    split_count_ = at::zeros({words}, like_.options().dtype(at::kInt).requires_grad(false));
  if (need > 0 && (!split_.defined() || split_.numel() < static_cast<int64_t>(need))) split_ = bytes(need, like_);
  check(lact_bmm_group_split_bf16(d, 2, need > 0 ? ptr(split_count_) : nullptr, need > 0 ? ptr(split_) : nullptr, need, status_, stream_),
        "lact_bmm_group_split_bf16");
}

void TokenBackward::apply(View w02, View w1, View q, View dO, int64_t n, View dW02, View dW1, bool accumulate, View dq) {
  const View dy = plane(a_, n, 2 * H_), hid = plane(b_, n, H_);
  // pre-activations y0, y2 = q w0^T, q w2^T and dh = dO w1 with the pointwise stage in their epilogue
  check(lact_fw_grad_pointwise(w02.p, w1.p, q.p, q.ld, q.bs, dO.p, dO.ld, dO.bs, nullptr, nullptr, nullptr, LACT_F32, 0, 1.0f,
                               const_cast<void*>(dy.p), const_cast<void*>(hid.p), B_, n, D_, H_, status_, stream_),
        "lact_fw_grad_pointwise");
  const lact_bmm_desc dw[2] = {product(dy, true, q, true, dW02, LACT_F32, accumulate, B_, 2 * H_, D_, n),
                               product(dO, true, hid, true, dW1, LACT_F32, accumulate, B_, D_, H_, n)};
  contraction(dw);
  const lact_bmm_desc dx = product(dy, false, w02, true, dq, LACT_BF16, false, B_, n, D_, 2 * H_);
  check(lact_bmm_group_bf16(&dx, 1, status_, stream_), "lact_bmm_group_bf16");
}

void TokenBackward::gradient(View w02, View w1, View k, View v, int64_t n, const void* const lr[3], int lr_dtype, int64_t lr_bs,
                             float w_scale, View g02, View g1, View dW02, View dW1, bool accumulate, View dk, View dv,
                             float* const glr[3], int64_t glr_bs, bool glr_add) {
  const View y = plane(a_, n, 2 * H_), dh = plane(b_, n, H_), gdy = plane(c_, n, 2 * H_), ghid = plane(d_, n, H_);
  const View gy = plane(e_, n, 2 * H_), gdh = plane(f_, n, H_), dyl = plane(g_, n, 2 * H_), hidl = plane(h_, n, H_);
  const lact_bmm_desc p0[2] = {product(k, false, w02, false, y, LACT_BF16, false, B_, n, 2 * H_, D_),
                               product(k, false, g02, false, gdy, LACT_BF16, false, B_, n, 2 * H_, D_)};
  check(lact_bmm_group_bf16(p0, 2, status_, stream_), "lact_bmm_group_bf16");
  const lact_bmm_desc p1[2] = {product(v, false, w1, true, dh, LACT_BF16, false, B_, n, H_, D_),
                               product(v, false, g1, true, ghid, LACT_BF16, false, B_, n, H_, D_)};
  check(lact_bmm_group_bf16(p1, 2, status_, stream_), "lact_bmm_group_bf16");
  auto m = [](View x) { return const_cast<void*>(x.p); };
  check(lact_fw_grad_bwd_pointwise(y.p, dh.p, gdy.p, ghid.p, lr[0], lr[1], lr[2], lr_dtype, w_scale, m(gy), m(gdh), m(dyl), m(hidl),
                                   glr[0], glr[1], glr[2], B_, n, H_, lr_bs, glr_bs, glr_add, stream_),
        "lact_fw_grad_bwd_pointwise");
  lact_bmm_desc p2[2] = {product(gy, false, w02, true, dk, LACT_BF16, false, B_, n, D_, 2 * H_),
                         product(gdh, false, w1, false, dv, LACT_BF16, false, B_, n, D_, H_)};
  plus(p2[0], dyl, false, g02, true);
  plus(p2[1], hidl, false, g1, false);
  check(lact_bmm_group_bf16(p2, 2, status_, stream_), "lact_bmm_group_bf16");
  const lact_bmm_desc p3[2] = {product(gy, true, k, true, dW02, LACT_F32, accumulate, B_, 2 * H_, D_, n),
                               product(v, true, gdh, true, dW1, LACT_F32, accumulate, B_, D_, H_, n)};
  contraction(p3);
}

namespace {

// Newton-Schulz of one group of gradient matrices as the backward needs it: result and trace
struct Orthogonal {
  int64_t nmat, R, C;
  const float* G;
  uint8_t* trace = nullptr;
  size_t trace_bytes = 0;
  Tensor keep, result_keep;   // trace / result this sweep computed itself
  const void* result = nullptr;  // bf16 [nmat][R][C]
};

class Sweep {
 public:
  Sweep(const Options& o, const Steps& st, const Tensor& like, int64_t B, int64_t L, int64_t D, int64_t H)
      : o_(o), st_(st), like_(like), B(B), L(L), D(D), H(H), n02(B * 2 * H * D), n1(B * D * H), status(status_word(like)),
        stream(stream_of(like)) {}

  // U = NS(G) from the trace the forward kept, or recomputed
  Orthogonal newton_schulz(const float* G, int64_t nmat, int64_t R, int64_t C, uint8_t* kept, size_t kept_bytes) {
    Orthogonal x{nmat, R, C, G};
    if (kept != nullptr) {
      size_t off = 0;
      check(lact_ns_trace_result_offset(nmat, R, C, o_.ns_steps, &off), "lact_ns_trace_result_offset");
      x.trace = kept; x.trace_bytes = kept_bytes;
      x.result = kept + off;
      return x;
    }
    x.result_keep = empty({nmat, R, C}, at::kBFloat16, like_);
    x.result = ptr(x.result_keep);
    size_t need = 0;
    if (o_.ns_steps == 0) {  // no iteration: the Frobenius normalisation alone
      check(lact_newton_schulz_workspace_bytes(nmat, R, C, &need), "lact_newton_schulz_workspace_bytes");
      const Tensor ws = bytes(need, like_);
      check(lact_newton_schulz(G, LACT_F32, ptr(x.result_keep), nmat, R, C, 0, 1, ptr(ws), ws.numel(), stream), "lact_newton_schulz");
      return x;
    }
    check(lact_ns_trace_bytes(nmat, R, C, o_.ns_steps, &need), "lact_ns_trace_bytes");
    x.keep = bytes(need, like_);
    x.trace = static_cast<uint8_t*>(ptr(x.keep)); x.trace_bytes = need;
    check(lact_ns_trace_fwd(G, LACT_F32, ptr(x.result_keep), nmat, R, C, o_.ns_steps, o_.const_coeffs, o_.gram_right, x.trace, need,
                            status, stream),
          "lact_ns_trace_fwd");
    return x;
  }

  // dG (fp32) of both groups from the bf16 gradients du of their results
  void newton_schulz_backward(Orthogonal* x, const Tensor* du, Tensor* dG) {
    const int64_t slices = lact_momentum_bwd_slices();
    Tensor part[2];
    lact_ns_bwd_group g[2];
    for (int i = 0; i < 2; ++i) {
      dG[i] = empty({x[i].nmat, x[i].R, x[i].C}, at::kFloat, like_);
      part[i] = empty({x[i].nmat * 2 * slices}, at::kFloat, like_);
      g[i] = lact_ns_bwd_group{ptr(du[i]), x[i].G, ptr(dG[i]), x[i].trace, x[i].trace_bytes, ptr(part[i]), x[i].nmat, x[i].R, x[i].C};
    }
    if (o_.ns_steps >= 1 && o_.ns_steps <= 5) {
      const int rc = lact_ns_trace_bwd_fused(g, 2, o_.ns_steps, o_.const_coeffs, o_.gram_right, status, stream);
      if (rc != LACT_ERR_CONFIG) return check(rc, "lact_ns_trace_bwd_fused");
    }
    for (int i = 0; i < 2; ++i) {
      if (o_.ns_steps == 0) dG[i].copy_(du[i].view(dG[i].sizes()));
      else
        check(lact_ns_trace_bwd(ptr(du[i]), ptr(dG[i]), x[i].nmat, x[i].R, x[i].C, o_.ns_steps, o_.const_coeffs, o_.gram_right,
                                x[i].trace, x[i].trace_bytes, status, stream),
              "lact_ns_trace_bwd");
      check(lact_ns_norm_bwd(x[i].G, ptr(dG[i]), ptr(part[i]), x[i].nmat, x[i].R * x[i].C, stream), "lact_ns_norm_bwd");
    }
  }

  const Options& o_;
  const Steps& st_;
  Tensor like_;
  int64_t B, L, D, H, n02, n1;
  StatusWord status;
  void* stream;
};

}  // namespace
}  // namespace lact_torch

#include "scan_sweep.inl"
