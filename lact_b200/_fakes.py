"""Shape-only implementations of the registered operators (tracing, `torch.compile`); registered once the operator library
has been loaded (`_lib.load_ops`)."""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib as L
from . import program as P

BF16, F32 = torch.bfloat16, torch.float32


_FAKES = {}   # every operator that this package calls


def _fake(name):
    def keep(fn):
        _FAKES[name] = fn
        return fn
    return keep


def register() -> None:
    """Raises ImportError, before it registers anything, if the loaded library lacks one of the operators."""
    missing = [name for name in _FAKES if not hasattr(torch.ops.lact_b200, name)]
    if missing:
        raise ImportError(f"{L.OPS_PATH} is older than this package (it has no {', '.join(missing)}): rebuild it with "
                          "`python -m lact_b200.build`")
    for name, fn in _FAKES.items():
        torch.library.register_fake("lact_b200::" + name, fn)


def ns_trace_bytes(B, Ltok, D, H, cfg) -> int:
    """Bytes of Newton-Schulz trace the training forward keeps per update (0: none)."""
    if not cfg[0]:
        return 0
    c = L.ScanConfig()
    c.B, c.L, c.D, c.H, c.out_len, c.act_dtype = B, Ltok, D, H, Ltok, L.LACT_BF16
    c.use_muon, c.ns_steps, c.ns_const_coeffs, c.ns_concat, c.ns_gram_right, c.renorm = (int(x) for x in cfg[:6])
    stride, off = C.c_size_t(0), C.c_size_t(0)
    return int(stride.value) if L.lib().lact_scan_ns_trace_bytes(C.byref(c), C.byref(stride), C.byref(off)) == 0 else 0


@_fake("scan_fwd")
def _(w0, w1, w2, q, k, v, lr0, lr1, lr2, momentum, m0, m1, m2, steps, cfg, w_scale):
    B, Ltok, D = k.shape
    H = w0.shape[1]
    state = lambda: [q.new_empty((B, H, D), dtype=F32), q.new_empty((B, D, H), dtype=F32), q.new_empty((B, H, D), dtype=F32)]
    outs = [q.new_empty((B, Ltok if cfg[10] < 0 else int(cfg[10]), D))]
    if cfg[13]:
        outs += state()
    if cfg[11]:
        outs += state()
    if cfg[12]:
        n_upd = sum(1 for i in range(0, len(steps), 4) if steps[i] == P.UPDATE)
        stride = ns_trace_bytes(B, Ltok, D, H, cfg)
        outs += [q.new_empty((max(n_upd, 1), 6 * B * D * H), dtype=F32),
                 q.new_empty((max(n_upd, 1) * stride if stride else 1,), dtype=torch.uint8),
                 q.new_empty((n_upd + 1, 3 * B * D * H), dtype=BF16)]
    return outs


@_fake("scan_bwd")
def _(w0, w1, w2, q, k, v, lr0, lr1, lr2, momentum, dump, trace, shadow, dO, gw0, gw1, gw2, steps, cfg, w_scale):
    outs = [t.new_empty(t.shape) for t in (w0, w1, w2, q, k, v, lr0, lr1, lr2)]
    return outs + [momentum.new_empty(momentum.shape)] if momentum is not None else outs


@_fake("swiglu_ffn_fwd")
def _(W0_W2, W1, X):
    return X.new_empty(X.shape)


@_fake("swiglu_ffn_bwd")
def _(W0_W2, W1, X, grad_out):
    return [t.new_empty(t.shape) for t in (W0_W2, W1, X)]


@_fake("fw_grads_fwd")
def _(W0_W2, W1, K, V, lr0, lr1, lr2):
    return [W0_W2.new_empty(W0_W2.shape), W1.new_empty(W1.shape)]


@_fake("fw_grads_bwd")
def _(W0_W2, W1, K, V, lr0, lr1, lr2, g02, g1):
    return [t.new_empty(t.shape) for t in (W0_W2, W1, K, V, lr0, lr1, lr2)]


@_fake("l2_norm_add_fwd")
def _(x, x_add, tgt_scale, eps, out_bf16):
    return x.new_empty(x.shape, dtype=BF16 if out_bf16 else F32)


@_fake("l2_norm_add_bwd")
def _(x, x_add, tgt_scale, dy, eps):
    return [t.new_empty(t.shape) for t in (x, x_add, tgt_scale)]


@_fake("swa_fwd")
def _(q, k, v, window, softmax_scale, seq_start=None):
    b, l, h, d = q.shape
    return [q.new_empty(q.shape), q.new_empty((b, h, l), dtype=F32)]


@_fake("swa_fwd_cache")
def _(q, k_cache, v_cache, k, v, softmax_scale):
    return q.new_empty(q.shape)


@_fake("swa_bwd")
def _(q, k, v, o, lse, dout, window, softmax_scale, seq_start=None):
    return [q.new_empty(q.shape), q.new_empty(k.shape), q.new_empty(k.shape)]


@_fake("seq_start")
def _(cu_seqlens, n_tokens):
    return cu_seqlens.new_empty((n_tokens,), dtype=torch.int32)


@_fake("qkv_prologue")
def _(xq, xk, xv, n_heads, silu, v_silu, cos, sin, rope_head_dim, offset, seq_start):
    b, s, nd = xq.shape
    return [xq.new_empty((b * n_heads, s, nd // n_heads)) for _ in range(3)]


@_fake("qkv_prologue_bwd")
def _(xq, xk, xv, dq, dk, dv, n_heads, silu, v_silu, cos, sin, rope_head_dim, offset, seq_start):
    return [xq.new_empty(xq.shape) for _ in range(3)]


@_fake("lr_prologue")
def _(proj, logits, n_heads, base_lr_inv):
    b, s, _ = proj.shape
    return [proj.new_empty((b * n_heads, s, 1), dtype=F32) for _ in range(4 if logits is not None else 3)]


@_fake("lr_prologue_bwd")
def _(proj, logits, g0, g1, g2, gm, n_heads, base_lr_inv):
    return [proj.new_empty(proj.shape)] + ([logits.new_empty(logits.shape)] if logits is not None else [])


@_fake("out_epilogue")
def _(fw_x, norm_weight, scale_proj, o, n_heads, eps):
    B, s, d = fw_x.shape
    return fw_x.new_empty((B // n_heads, s, n_heads * d))


@_fake("out_epilogue_bwd")
def _(fw_x, norm_weight, scale_proj, dout, n_heads, eps):
    outs = [fw_x.new_empty(fw_x.shape), norm_weight.new_empty(norm_weight.shape, dtype=F32)]
    return outs + [scale_proj.new_empty(scale_proj.shape)] if scale_proj is not None else outs
