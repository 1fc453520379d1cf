// What the forward and the backward of the recurrence share: options as the operators pass them, sizes, step lists.
#pragma once
#include "common.h"

namespace lact_torch {

// cfg of lact_b200::scan_fwd / scan_bwd, in order
struct Options {
  bool muon;
  int32_t ns_steps;
  bool const_coeffs, concat, gram_right;
  int32_t renorm;
  bool prenorm, prenorm_bf16, overwrite, detach_norms;
  int64_t out_len;  // -1: as many as there are tokens
  bool return_momentum, save, return_state;
  static constexpr size_t kFields = 14;
  explicit Options(at::IntArrayRef c) {
    TORCH_CHECK_VALUE(c.size() == kFields, "cfg must have ", kFields, " entries");
    muon = c[0]; ns_steps = static_cast<int32_t>(c[1]); const_coeffs = c[2]; concat = c[3]; gram_right = c[4];
    renorm = static_cast<int32_t>(c[5]); prenorm = c[6]; prenorm_bf16 = c[7]; overwrite = c[8]; detach_norms = c[9];
    out_len = c[10]; return_momentum = c[11]; save = c[12]; return_state = c[13];
  }
};

struct Steps {
  std::vector<int32_t> kind;
  std::vector<int64_t> start, end, out;
  int32_t n = 0, updates = 0;
  explicit Steps(at::IntArrayRef flat) {
    TORCH_CHECK_VALUE(flat.size() % 4 == 0, "steps are (kind, start, end, out_start) quadruples");
    n = static_cast<int32_t>(flat.size() / 4);
    kind.resize(n); start.resize(n); end.resize(n); out.resize(n);
    for (int32_t i = 0; i < n; ++i) {
      kind[i] = static_cast<int32_t>(flat[4 * i]);
      start[i] = flat[4 * i + 1]; end[i] = flat[4 * i + 2]; out[i] = flat[4 * i + 3];
      updates += kind[i] == kUpdate;
    }
  }
  // Token ranges of [0, total) that no step of `which` covers (`by_out`: ranges of the output instead of the input).
  std::vector<std::pair<int64_t, int64_t>> gaps(Step which, int64_t total, bool by_out) const {
    std::vector<std::pair<int64_t, int64_t>> r, g;
    for (int32_t i = 0; i < n; ++i)
      if (kind[i] == which && end[i] > start[i]) {
        const int64_t s = by_out ? out[i] : start[i];
        r.emplace_back(s, s + end[i] - start[i]);
      }
    std::sort(r.begin(), r.end());
    int64_t at = 0;
    for (auto& [s, e] : r) {
      if (s > at) g.emplace_back(at, s);
      at = std::max(at, e);
    }
    if (at < total) g.emplace_back(at, total);
    return g;
  }
};

// Sizes and options as the C ABI takes them (activations bf16, no strides): what the layout queries need.
inline lact_scan_config base_config(const Options& o, int64_t B, int64_t L, int64_t D, int64_t H) {
  lact_scan_config c;
  std::memset(&c, 0, sizeof(c));
  c.B = B; c.L = L; c.D = D; c.H = H;
  c.out_len = o.out_len < 0 ? L : o.out_len;
  c.act_dtype = LACT_BF16;
  c.use_muon = o.muon; c.ns_steps = o.ns_steps; c.ns_const_coeffs = o.const_coeffs; c.ns_concat = o.concat;
  c.ns_gram_right = o.gram_right; c.renorm = o.renorm; c.prenorm = o.prenorm; c.prenorm_bf16 = o.prenorm_bf16;
  c.overwrite_quirk = o.overwrite;
  return c;
}

// Bytes of Newton-Schulz trace the training forward keeps per update and the offset of the w1 group's part, or zeros
// when this configuration keeps none (Muon off, more than five iterations).
inline std::pair<size_t, size_t> trace_layout(const Options& o, int64_t B, int64_t L, int64_t D, int64_t H) {
  size_t stride = 0, off = 0;
  if (!o.muon) return {0, 0};
  const lact_scan_config c = base_config(o, B, L, D, H);
  if (lact_scan_ns_trace_bytes(&c, &stride, &off) != LACT_OK) return {0, 0};
  return {stride, off};
}

// fp32 elements of one slot of the training state: [w0w2 | w1 | g0g2 | g1]
inline int64_t state_elems(int64_t B, int64_t D, int64_t H) { return 2 * B * 3 * D * H; }

}  // namespace lact_torch
