// The reverse sweep itself (included by scan_bwd.cpp).
namespace lact_torch {
namespace {

std::vector<Tensor> scan_bwd(const Tensor& w0, const Tensor& w1, const Tensor& w2, const Tensor& q_, const Tensor& k_,
                             const Tensor& v_, const Tensor& lr0, const Tensor& lr1, const Tensor& lr2, const OptTensor& momentum,
                             const Tensor& dump, const Tensor& trace, const Tensor& shadow, const Tensor& dO_, const OptTensor& gw0,
                             const OptTensor& gw1, const OptTensor& gw2, at::IntArrayRef steps_, at::IntArrayRef cfg_,
                             double w_scale) {
  const c10::cuda::CUDAGuard guard(k_.device());
  const Options o(cfg_);
  const Steps st(steps_);
  const Tensor q = aligned(q_), k = aligned(k_), v = aligned(v_), dO = aligned(dO_.to(at::kBFloat16));
  const int64_t B = k.size(0), L = k.size(1), D = k.size(2), H = w0.size(1);
  Sweep sw(o, st, k, B, L, D, H);
  const int64_t n02 = sw.n02, n1 = sw.n1;
  void* const stream = sw.stream;
  const auto F = at::kFloat, BF = at::kBFloat16;
  const bool has_mom = given(momentum), overwrite = o.overwrite && o.muon;

  // state the forward kept: fp32 weights and gradients per update, bf16 weights per slot, Newton-Schulz traces
  float* const state = dump.data_ptr<float>();
  auto slot = [&](int u) { return state + static_cast<int64_t>(u) * 2 * (n02 + n1); };
  auto G02 = [&](int u) { return slot(u) + n02 + n1; };
  auto G1 = [&](int u) { return slot(u) + 2 * n02 + n1; };
  auto W02b = [&](int u) { return View(static_cast<at::BFloat16*>(ptr(shadow)) + u * (n02 + n1), D, 2 * H * D); };
  auto W1b = [&](int u) { return View(static_cast<at::BFloat16*>(ptr(shadow)) + u * (n02 + n1) + n02, H, D * H); };
  const auto [tr_stride, tr_off] = trace.numel() > 1 ? trace_layout(o, B, L, D, H) : std::pair<size_t, size_t>{0, 0};
  auto kept = [&](int u, int group) -> uint8_t* {
    return tr_stride ? static_cast<uint8_t*>(ptr(trace)) + u * tr_stride + (group ? tr_off : 0) : nullptr;
  };
  auto kept_bytes = [&](int group) { return group ? tr_stride - tr_off : tr_off; };
  const int64_t m02 = o.concat ? B : 2 * B, r02 = o.concat ? 2 * H : H;
  auto wrap = [&](float* p, at::IntArrayRef shape) { return at::from_blob(p, shape, k.options().dtype(F).requires_grad(false)); };

  auto vec = [&](const Tensor& t) { return (t.dim() == 3 ? t.select(2, 0) : t).contiguous(); };
  Tensor lrv[3] = {vec(lr0), vec(lr1), vec(lr2)};
  for (Tensor& t : lrv)
    if (t.scalar_type() != lrv[0].scalar_type() || (t.scalar_type() != F && t.scalar_type() != BF)) {
      for (Tensor& x : lrv) x = x.to(F);
      break;
    }
  const int64_t lr_esz = lrv[0].element_size();

  // target row norms (of the initial weights) and their gradients
  Tensor n0_02, n0_1, dn02, dn1;
  if (st.updates > 0) {
    n0_02 = at::linalg_vector_norm(wrap(slot(0), {B, 2 * H, D}), 2, {2});
    n0_1 = at::linalg_vector_norm(wrap(slot(0) + n02, {B, D, H}), 2, {2});
    dn02 = at::zeros({B, 2 * H}, n0_02.options());
    dn1 = at::zeros({B, D}, n0_02.options());
  }

  // momentum factors and gate gradients per update
  Tensor beta, dbeta;
  std::vector<int64_t> us, ue;
  for (int i = 0; i < st.n; ++i)
    if (st.kind[i] == kUpdate) { us.push_back(st.start[i]); ue.push_back(st.end[i]); }
  const int64_t slices = lact_momentum_bwd_slices();
  if (has_mom && st.updates > 0) {
    Tensor mv = vec(*momentum);
    if (mv.scalar_type() != F && mv.scalar_type() != BF) mv = mv.to(F);
    beta = empty({st.updates, B}, F, k);
    check(lact_momentum_means(ptr(mv), dtype_code(mv), B, L, st.updates, us.data(), ue.data(), beta.data_ptr<float>(), stream),
          "lact_momentum_means");
    dbeta = empty({st.updates, B, slices}, F, k);
    dbeta.select(0, 0).zero_();  // nothing precedes the first update
  }

  // pre-norm: un-normalised master weights before each update, Wm_0 = W_0, Wm_{u+1} = Wm_u + U_u
  std::vector<Tensor> masters02, masters1;
  if (o.prenorm && st.updates > 0) {
    masters02.push_back(wrap(slot(0), {B, 2 * H, D}));
    masters1.push_back(wrap(slot(0) + n02, {B, D, H}));
    for (int u = 0; u + 1 < st.updates; ++u) {
      Tensor u02 = wrap(G02(u), {B, 2 * H, D}), u1 = wrap(G1(u), {B, D, H});
      if (o.muon) {
        const Orthogonal x = sw.newton_schulz(G02(u), m02, r02, D, kept(u, 0), kept_bytes(0));
        const Orthogonal y = sw.newton_schulz(G1(u), B, D, H, kept(u, 1), kept_bytes(1));
        u02 = at::from_blob(const_cast<void*>(x.result), {B, 2 * H, D}, k.options().dtype(BF).requires_grad(false));
        u1 = at::from_blob(const_cast<void*>(y.result), {B, D, H}, k.options().dtype(BF).requires_grad(false));
        masters02.push_back(at::add(masters02.back(), u02));
        masters1.push_back(at::add(masters1.back(), u1));
        continue;
      }
      masters02.push_back(at::add(masters02.back(), u02));
      masters1.push_back(at::add(masters1.back(), u1));
    }
  }

  // gradient w.r.t. the weights the later steps computed with; `fresh`: nothing has been added to it yet
  Tensor dW02 = empty({B, 2 * H, D}, F, k), dW1 = empty({B, D, H}, F, k);
  bool fresh = true;
  if (given(gw0) || given(gw1) || given(gw2)) {  // cotangents of the returned final weights
    auto put = [](Tensor dst, const OptTensor& g) { if (given(g)) dst.copy_(*g); else dst.zero_(); };
    put(dW02.narrow(1, 0, H), gw0);
    put(dW02.narrow(1, H, H), gw2);
    put(dW1, gw1);
    fresh = false;
  }
  Tensor dWm02, dWm1;  // pre-norm: w.r.t. the master weights after the current update
  Tensor dM02, dM1;    // w.r.t. the momentum state after the current update

  Tensor dq = empty({B, L, D}, BF, k), dk = empty({B, L, D}, BF, k), dv = empty({B, L, D}, BF, k), dlr[3];
  // every token range is written in place by the first step that has a gradient for it; the others are zero
  for (auto& [s, e] : st.gaps(kApply, L, false)) dq.narrow(1, s, e - s).zero_();
  const auto upd_gaps = st.gaps(kUpdate, L, false);
  for (Tensor& t : dlr) t = empty({B, L}, F, k);
  for (auto& [s, e] : upd_gaps) {
    dk.narrow(1, s, e - s).zero_();
    dv.narrow(1, s, e - s).zero_();
    for (Tensor& t : dlr) t.narrow(1, s, e - s).zero_();
  }
  // (in part, if ranges overlap: what no step has written yet of a range that is added to is zeroed first)
  using Ranges = std::vector<std::pair<int64_t, int64_t>>;
  Ranges q_done, kv_done, o_done;
  // Whether [s, e) has been written nowhere; otherwise `missing` receives the parts of it that have not.
  auto first = [](Ranges& done, int64_t s, int64_t e, Ranges& missing) {
    bool ok = true;
    missing.assign(1, {s, e});
    for (auto& [a, b] : done) {
      if (e <= a || s >= b) continue;
      ok = false;
      Ranges left;
      for (auto& [x, y] : missing) {
        if (x < std::min(y, a)) left.emplace_back(x, std::min(y, a));
        if (std::max(x, b) < y) left.emplace_back(std::max(x, b), y);
      }
      missing.swap(left);
    }
    done.emplace_back(s, e);
    return ok;
  };
  Ranges missing, kept_out;

  TokenBackward tok(B, D, H, k, sw.status, stream);
  int cnt = st.updates;
  for (int i = st.n - 1; i >= 0; --i) {
    const int64_t s = st.start[i], e = st.end[i], n = e - s;
    if (n <= 0) continue;
    if (st.kind[i] == kApply) {
      // (of outputs that a later step writes again, only the last has a gradient)
      const int64_t at = st.out[i];
      Tensor last;
      View go = tokens(dO, at);
      if (!first(o_done, at, at + n, kept_out)) {
        last = at::zeros({B, n, D}, dO.options());
        for (auto& [a, b] : kept_out) last.narrow(1, a - at, b - a).copy_(dO.narrow(1, a, b - a));
        go = View(last);
      }
      const bool own = first(q_done, s, e, missing);
      if (last.defined() && kept_out.empty()) {
        for (auto& [a, b] : missing) dq.narrow(1, a, b - a).zero_();
        continue;
      }
      Tensor tmp = own ? Tensor() : empty({B, n, D}, BF, k);
      tok.apply(W02b(cnt), W1b(cnt), tokens(q, s), go, n, View(dW02), View(dW1), !fresh, own ? tokens(dq, s) : View(tmp));
      fresh = false;
      if (!own) {
        for (auto& [a, b] : missing) dq.narrow(1, a, b - a).zero_();
        dq.narrow(1, s, n).add_(tmp);
      }
      continue;
    }
    const int u = --cnt;
    if (fresh) { dW02.zero_(); dW1.zero_(); }
    Orthogonal ns[2];
    if (o.muon) {
      ns[0] = sw.newton_schulz(G02(u), m02, r02, D, kept(u, 0), kept_bytes(0));
      ns[1] = sw.newton_schulz(G1(u), B, D, H, kept(u, 1), kept_bytes(1));
    }
    // renorm backward: dWn = gradient w.r.t. (base + update); base = W_u, the master copy (pre-norm), or the gradient
    // itself (bidirectional overwrite)
    const float* base02 = o.prenorm ? masters02[u].data_ptr<float>() : (overwrite ? G02(u) : slot(u));
    const float* base1 = o.prenorm ? masters1[u].data_ptr<float>() : (overwrite ? G1(u) : slot(u) + n02);
    const bool carry_in = o.prenorm && dWm02.defined(), want_b = o.muon && !carry_in;
    Tensor dWn02 = empty({B, 2 * H, D}, F, k), dWn1 = empty({B, D, H}, F, k), dub[2];
    if (want_b) { dub[0] = empty({B, 2 * H, D}, BF, k); dub[1] = empty({B, D, H}, BF, k); }
    check(lact_renorm_bwd(base02, o.muon ? ns[0].result : static_cast<const void*>(G02(u)), o.muon ? LACT_BF16 : LACT_F32, ptr(n0_02),
                          ptr(dW02), ptr(dWn02), want_b ? ptr(dub[0]) : nullptr, ptr(dn02), B * 2 * H, D, o.renorm, stream),
          "lact_renorm_bwd");
    check(lact_renorm_bwd(base1, o.muon ? ns[1].result : static_cast<const void*>(G1(u)), o.muon ? LACT_BF16 : LACT_F32, ptr(n0_1),
                          ptr(dW1), ptr(dWn1), want_b ? ptr(dub[1]) : nullptr, ptr(dn1), B * D, H, o.renorm, stream),
          "lact_renorm_bwd");
    if (carry_in) {
      dWn02.add_(dWm02);
      dWn1.add_(dWm1);
    }
    Tensor dG[2] = {dWn02, dWn1};
    if (o.muon) {
      if (!want_b) { dub[0] = dWn02.to(BF); dub[1] = dWn1.to(BF); }
      sw.newton_schulz_backward(ns, dub, dG);
      if (overwrite) {
        dG[0].view({B, 2 * H, D}).add_(dWn02);
        dG[1].add_(dWn1);
      }
    }
    if (o.prenorm) { dWm02 = dWn02; dWm1 = dWn1; }
    if (o.prenorm || overwrite) {  // the weights update u computed with receive gradient only from its own steps
      dW02 = empty({B, 2 * H, D}, F, k); dW1 = empty({B, D, H}, F, k);
      fresh = true;
    } else {
      dW02 = dWn02; dW1 = dWn1;
      fresh = false;
    }
    // momentum step: what arrives from the next update's momentum state, the gate's gradient, the share that goes on to
    // the previous update, and the bf16 copies the contractions below read
    Tensor g02b = empty({B, 2 * H, D}, BF, k), g1b = empty({B, D, H}, BF, k);
    const bool add_carry = dM02.defined();
    if (has_mom && !add_carry) { dM02 = empty({B, 2 * H, D}, F, k); dM1 = empty({B, D, H}, F, k); }
    const bool prev = has_mom && u > 0;
    check(lact_momentum_bwd(ptr(dG[0]), ptr(dG[1]), has_mom ? ptr(dM02) : nullptr, has_mom ? ptr(dM1) : nullptr,
                            prev ? G02(u - 1) : nullptr, prev ? G1(u - 1) : nullptr, ptr(g02b), ptr(g1b),
                            has_mom ? beta.data_ptr<float>() + static_cast<int64_t>(u) * B : nullptr,
                            prev ? dbeta.data_ptr<float>() + static_cast<int64_t>(u) * B * slices : nullptr, B, 2 * H * D, D * H,
                            add_carry, stream),
          "lact_momentum_bwd");
    const void* lr[3];
    for (int j = 0; j < 3; ++j) lr[j] = static_cast<const uint8_t*>(ptr(lrv[j])) + s * lr_esz;
    float* glr[3];
    for (int j = 0; j < 3; ++j) glr[j] = dlr[j].data_ptr<float>() + s;
    const bool own = first(kv_done, s, e, missing);
    Tensor tk, tv;
    if (!own) {
      tk = empty({B, n, D}, BF, k);
      tv = empty({B, n, D}, BF, k);
      for (auto& [a, b] : missing) {
        dk.narrow(1, a, b - a).zero_();
        dv.narrow(1, a, b - a).zero_();
        for (Tensor& t : dlr) t.narrow(1, a, b - a).zero_();
      }
    }
    tok.gradient(W02b(u), W1b(u), tokens(k, s), tokens(v, s), n, lr, dtype_code(lrv[0]), L, static_cast<float>(w_scale), View(g02b),
                 View(g1b), View(dW02), View(dW1), !fresh, own ? tokens(dk, s) : View(tk), own ? tokens(dv, s) : View(tv), glr, L,
                 !own);
    fresh = false;
    if (!own) {
      dk.narrow(1, s, n).add_(tk);
      dv.narrow(1, s, n).add_(tv);
    }
  }
  if (fresh) { dW02.zero_(); dW1.zero_(); }

  // W_0 is both the first master and the first compute copy; its row norms are the targets unless detached
  const bool norms = !o.detach_norms && st.updates > 0;
  const bool lowp = w0.scalar_type() == BF && w1.scalar_type() == BF && w2.scalar_type() == BF;
  const auto wt = lowp ? BF : F;
  Tensor dw0 = empty({B, H, D}, wt, k), dw1 = empty({B, D, H}, wt, k), dw2 = empty({B, H, D}, wt, k);
  auto fp = [](const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; };
  check(lact_weight_grad(fp(dW02), fp(dW1), fp(dWm02), fp(dWm1), norms ? fp(dn02) : nullptr, norms ? fp(dn1) : nullptr, fp(n0_02),
                         fp(n0_1), st.updates > 0 ? slot(0) : nullptr, st.updates > 0 ? slot(0) + n02 : nullptr, ptr(dw0), ptr(dw1),
                         ptr(dw2), lowp ? LACT_BF16 : LACT_F32, B, D, H, stream),
        "lact_weight_grad");
  auto like = [](const Tensor& g, const Tensor& ref) { return g.view(ref.sizes()).to(ref.scalar_type()); };
  std::vector<Tensor> r{dw0.to(w0.scalar_type()), dw1.to(w1.scalar_type()), dw2.to(w2.scalar_type()), dq.to(q_.scalar_type()),
                        dk.to(k_.scalar_type()), dv.to(v_.scalar_type()), like(dlr[0], lr0), like(dlr[1], lr1), like(dlr[2], lr2)};
  if (has_mom) {
    // (bf16 only where one launch writes it: later ones add to what is there)
    const bool mb = momentum->scalar_type() == BF && st.updates <= LACT_GATE_GRAD_UPDATES;
    Tensor dm = empty({B, L}, mb ? BF : F, k);
    if (st.updates > 0)
      check(lact_momentum_gate_grad(dbeta.data_ptr<float>(), B, L, st.updates, us.data(), ue.data(), ptr(dm), mb ? LACT_BF16 : LACT_F32,
                                    stream),
            "lact_momentum_gate_grad");
    else dm.zero_();
    r.push_back(like(dm, *momentum));
  }
  settle(k);
  return r;
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(lact_b200, m) {
  m.def("scan_bwd(Tensor w0, Tensor w1, Tensor w2, Tensor q, Tensor k, Tensor v, Tensor lr0, Tensor lr1, Tensor lr2, "
        "Tensor? momentum, Tensor dump, Tensor trace, Tensor shadow, Tensor dO, Tensor? gw0, Tensor? gw1, Tensor? gw2, int[] steps, "
        "int[] cfg, float w_scale) -> Tensor[]");
}
TORCH_LIBRARY_IMPL(lact_b200, CUDA, m) { m.impl("scan_bwd", &scan_bwd); }
TORCH_LIBRARY_IMPL(lact_b200, Autograd, m) {
  m.impl("scan_bwd", torch::autograd::autogradNotImplementedFallback());
}

}  // namespace lact_torch
