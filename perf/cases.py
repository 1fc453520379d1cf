"""The calls this package is used for, as measurable cases.

`listed()` are fixed cases, `draw()` gives others of the same ranges; a case is a dict of plain values whose "kind"
says which public entry points it calls.  `prepare()` makes what a caller holds before the call (inputs on the GPU,
weights, momentum state, rotary tables), `run()` is one call (forward, or forward and backward) and returns everything
it computes, `work()` the bytes and operations it cannot do without, `tolerance()` how far two correct implementations
of the same precision may differ.

Inputs: q, k, v ~ N(0, 1) with q, k normalised per token, fast weights ~ N(0, 1 / fan-in), learning rates
softplus(N(-2, 1)), momentum gates sigmoid(N(0, 1)), gradients of outputs ~ N(0, 1).
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import lact_b200 as lb
from lact_b200 import layer_ops as lo

BF16, F32 = torch.bfloat16, torch.float32


# ---------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # a language model's layer at its usual size: 8 sequences of 32768 tokens, 4 heads of 384 (prefill / evaluation)
        dict(name="llm_forward", kind="causal", form="post_fused", units=32, tokens=32768, d=384, h=384, chunk=2048,
             muon=True, momentum=True, lr="bf16", train=False),
        # the same layer in training: forward and gradients of every input
        dict(name="llm_train", kind="causal", form="post_fused", units=32, tokens=32768, d=384, h=384, chunk=2048,
             muon=True, momentum=True, lr="bf16", train=True),
        # one prompt of a length no chunk divides, pre-norm layer (one sequence, 4 heads, or one GPU's share of a batch)
        dict(name="llm_prompt", kind="causal", form="pre_fused", units=4, tokens=5003, d=384, h=384, chunk=2048,
             muon=True, momentum=True, lr="f32", train=False),
        # generation between two updates of the fast weights: a few new tokens through the current weights
        dict(name="llm_decode", kind="ffn", units=4, tokens=16, d=384, h=384),
        # the minimal bidirectional layer as its module runs it, fp32 activations
        dict(name="bidirectional_fp32", kind="bidirectional", units=4, tokens=4096, d=192, h=192, muon=True, dtype="f32"),
        # novel-view synthesis, inference: one update on 48 input views, applied to 4 target views
        dict(name="nvs_render", kind="nvs", units=16, d=192, h=192, inputs=49152, targets=4096, all_tokens=False,
             muon_steps=5, train=False),
        # novel-view synthesis, training: 8 input views and 4 target views, every token read back
        dict(name="nvs_train", kind="nvs", units=8, d=192, h=192, inputs=8192, targets=4096, all_tokens=True,
             muon_steps=5, train=True),
        # autoregressive video over a whole clip: 21 frames of 1560 tokens, one update per frame
        dict(name="video_clip", kind="video", units=12, d=128, h=256, frame=1560, frames=21, spacing=1, muon=True,
             momentum=True, train=False),
        # autoregressive video, generation: one finished frame updates the state that the next frame starts from
        dict(name="video_step", kind="video_step", units=12, d=128, h=256, frame=1560, update=True, muon=True),
        # the attention half of a hybrid layer in training: causal window of 2048
        dict(name="window_train", kind="window", batch=2, tokens=32768, heads=12, d=128, window=2048, sequences=1, train=True),
        # the attention half of a video layer in generation: one frame over a cache of two frames
        dict(name="cache_attention", kind="cache", batch=1, tokens=1560, cached=3120, heads=12, d=128),
        # the passes around the recurrence in a hybrid layer's training step: heads, SiLU, norms, rotation, gates
        dict(name="layer_passes_train", kind="layer", batch=2, tokens=8192, heads=4, d=384, rotary=128, train=True),
    ]


def _log(rng, lo_, hi, step=1):
    """An integer of [lo_, hi], spread over the logarithm, on a grid of `step`."""
    v = math.exp(rng.uniform(math.log(lo_), math.log(hi)))
    return max(lo_, min(hi, int(round(v / step)) * step))


def _tokens(rng, lo_, hi):
    """A token count: a multiple of 128 as often as not, else whatever comes."""
    return _log(rng, lo_, hi, 128 if lo_ >= 128 and rng.random() < 0.5 else 1)


_LLM_HEAD = ((384, 384), (384, 384), (256, 256), (512, 512), (192, 192), (128, 256))
_MUON_TRAIN_HEAD = ((384, 384), (384, 384), (192, 192), (128, 256))   # head sizes the Newton-Schulz backward takes


def draw(rng):
    kind = rng.choice(("causal", "causal", "causal", "ffn", "bidirectional", "nvs", "nvs", "video", "video_step", "window",
                       "cache", "layer"))
    if kind == "causal":
        muon, train = rng.random() < 0.6, rng.random() < 0.4
        d, h = rng.choice(_MUON_TRAIN_HEAD if muon and train else _LLM_HEAD)
        units = rng.choice((1, 2, 3, 4, 6, 8, 12, 16, 24, 32))
        chunk = rng.choice((512, 1024, 2048, 2048, 4096, 1000))
        # at most 16 chunks, and no more tokens in all than the largest listed case
        most = max(600, min(16 * chunk, int(32 * 32768 * (384 * 384) / (d * h)) // units))
        return dict(kind=kind, form=rng.choice(("post_fused", "pre_fused", "post", "pre")), units=units,
                    tokens=_tokens(rng, min(512, most), min(32768, most)), d=d, h=h, chunk=chunk,
                    muon=muon, momentum=rng.random() < 0.7, lr=rng.choice(("bf16", "f32")), train=train)
    if kind == "ffn":
        d, h = rng.choice(_LLM_HEAD)
        return dict(kind=kind, units=rng.choice((1, 2, 4, 8, 16, 32)), tokens=_log(rng, 1, 2048), d=d, h=h)
    if kind == "bidirectional":
        dtype = rng.choice(("bf16", "bf16", "f32"))
        d, h = rng.choice(((192, 192), (128, 128), (256, 256), (64, 128)))
        return dict(kind=kind, units=rng.choice((2, 4, 8, 16)), tokens=_tokens(rng, 256, 8192 if dtype == "f32" else 32768),
                    d=d, h=h, muon=rng.random() < 0.6, dtype=dtype)
    if kind == "nvs":
        train = rng.random() < 0.5
        d, h = rng.choice(((192, 192), (192, 192), (128, 128), (64, 128)) if train else ((192, 192), (192, 192), (256, 256), (128, 128)))
        return dict(kind=kind, units=rng.choice((4, 8, 12, 16)), d=d, h=h, inputs=_tokens(rng, 1024, 16384 if train else 49152),
                    targets=_tokens(rng, 256, 8192), all_tokens=rng.random() < 0.5, muon_steps=rng.choice((5, 5, 3, 1)),
                    train=train)
    if kind == "video":
        return dict(kind=kind, units=rng.choice((6, 12, 12, 24)), d=128, h=rng.choice((128, 256, 256)), frame=_tokens(rng, 384, 1560),
                    frames=rng.randint(2, 21), spacing=rng.choice((1, 1, 2)), muon=rng.random() < 0.6,
                    momentum=rng.random() < 0.6, train=rng.random() < 0.3)
    if kind == "video_step":
        return dict(kind=kind, units=rng.choice((6, 12, 12, 24)), d=128, h=rng.choice((128, 256, 256)), frame=_tokens(rng, 200, 4680),
                    update=rng.random() < 0.6, muon=rng.random() < 0.7)
    if kind == "window":
        d = rng.choice((64, 128, 128))
        tokens = _tokens(rng, 256, 32768)
        return dict(kind=kind, batch=rng.choice((1, 2)), tokens=tokens, heads=rng.choice((4, 8, 12)), d=d,
                    window=rng.choice((256, 512, 1024, 2048, 2048)),
                    sequences=rng.choice((1, 1, 2, 5)), train=rng.random() < 0.6) | ({} if tokens >= 1024 else {"sequences": 1})
    if kind == "cache":
        return dict(kind=kind, batch=rng.choice((1, 1, 2)), tokens=_tokens(rng, 100, 4680), cached=_log(rng, 1, 12480),
                    heads=rng.choice((4, 8, 12, 16)), d=rng.choice((64, 128, 128)))
    d = rng.choice((64, 128, 192, 256, 384, 512))
    return dict(kind=kind, batch=rng.choice((1, 2, 4)), tokens=_tokens(rng, 128, 8192), heads=rng.choice((2, 4, 6)), d=d,
                rotary=rng.choice((0, 64, 128)) if d % 128 == 0 else rng.choice((0, 64)), train=rng.random() < 0.6)


# ---------------------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rows(g, *shape, dtype=BF16, unit=False):
    x = torch.randn(*shape, device="cuda", generator=g)
    if unit:
        x /= x.norm(dim=-1, keepdim=True)
    return x.to(dtype)


def _recurrence(c, seed, tokens, dtype=BF16, lr=F32, momentum=False):
    """The arguments of a chunk driver in the order its signature has them, and the momentum gate."""
    g = _generator(seed)
    b, d, h = c["units"], c["d"], c["h"]
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    w = [rn(b, h, d) / d ** 0.5, rn(b, d, h) / h ** 0.5, rn(b, h, d) / d ** 0.5]
    qkv = [_rows(g, b, tokens, d, dtype=dtype, unit=i < 2) for i in range(3)]
    lrs = [F.softplus(rn(b, tokens, 1) - 2.0).to(lr) for _ in range(3)]
    gate = torch.sigmoid(rn(b, tokens, 1)) if momentum else None
    return w + qkv + lrs, gate, g


def _leaves(tensors):
    return [None if t is None else t.detach().requires_grad_(True) for t in tensors]


_CAUSAL = {
    "post_fused": lb.postnorm_block_causal_lact_swiglu_fused_kernel_triton,
    "pre_fused": lb.prenorm_block_causal_lact_swiglu_fused_kernel_triton,
    "post": lb.block_causal_lact_swiglu,
    "pre": lb.prenorm_block_causal_lact_swiglu,
}


def _video_length(c):
    # tokens before the first update, then `frames` strides
    return (c["spacing"] - 1) * c["frame"] + c["frames"] * c["spacing"] * c["frame"]


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "causal":
        args, gate, g = _recurrence(c, seed, c["tokens"], lr=BF16 if c["lr"] == "bf16" else F32, momentum=c["momentum"])
        if not c["train"]:
            return dict(case=c, args=args, gate=gate)
        leaves = _leaves(args + [gate])
        return dict(case=c, args=leaves[:9], gate=leaves[9], dout=_rows(g, c["units"], c["tokens"], c["d"]))
    if kind == "ffn":
        g = _generator(seed)
        b, d, h = c["units"], c["d"], c["h"]
        w02 = torch.randn(b, 2 * h, d, device="cuda", generator=g) / d ** 0.5
        w1 = torch.randn(b, d, h, device="cuda", generator=g) / h ** 0.5
        return dict(case=c, w02=w02.to(BF16), w1=w1.to(BF16), x=_rows(g, b, c["tokens"], d, unit=True))
    if kind == "bidirectional":
        args, _, _ = _recurrence(c, seed, c["tokens"], dtype=BF16 if c["dtype"] == "bf16" else F32)
        return dict(case=c, args=args)
    if kind == "nvs":
        n = c["inputs"] + c["targets"]
        args, _, g = _recurrence(c, seed, n)
        for i in range(3):   # this layer keeps its weights [b, d, dh], [b, dh, d], [b, d, dh]
            args[i] = args[i].transpose(1, 2).contiguous()
        read = (0, n) if c["all_tokens"] else (c["inputs"], n)
        order = [lb.TTTOperator(0, c["inputs"], True, False), lb.TTTOperator(*read, False, True)]
        if not c["train"]:
            return dict(case=c, args=args, order=order)
        return dict(case=c, args=_leaves(args), order=order, dout=_rows(g, c["units"], read[1] - read[0], c["d"]))
    if kind == "video":
        n = _video_length(c)
        args, gate, g = _recurrence(c, seed, n, momentum=c["momentum"])
        if not c["train"]:
            return dict(case=c, args=args, gate=gate)
        leaves = _leaves(args + [gate])
        return dict(case=c, args=leaves[:9], gate=leaves[9], dout=_rows(g, c["units"], n, c["d"]))
    if kind == "video_step":
        args, gate, g = _recurrence(c, seed, c["frame"], momentum=True)
        m = [torch.randn(w.shape, device="cuda", generator=g) for w in args[:3]]   # momentum left by the frames before
        return dict(case=c, args=args, gate=gate, m=m)
    if kind == "window":
        g = _generator(seed)
        b, n, h, d, s = c["batch"], c["tokens"], c["heads"], c["d"], c["sequences"]
        if s > 1:   # sequences packed back to back: one batch entry
            b = 1
        qkv = _rows(g, b, n, 3 * h * d).view(b, n, 3, h, d)   # a fused projection; q, k, v are views of it
        q, k, v = (qkv[:, :, i] for i in range(3))
        cu = torch.tensor([round(i * n / s) - (1 if 0 < i < s and i % 2 else 0) for i in range(s + 1)], dtype=torch.int32,
                          device="cuda") if s > 1 else None
        if c["train"]:
            q, k, v = _leaves((q, k, v))
        return dict(case=c, q=q, k=k, v=v, cu=cu, dout=_rows(g, b, n, h, d) if c["train"] else None)
    if kind == "cache":
        g = _generator(seed)
        b, h, d = c["batch"], c["heads"], c["d"]
        q, k, v = (_rows(g, b, c["tokens"], h, d) for _ in range(3))
        return dict(case=c, q=q, k=k, v=v, cache=_rows(g, 2 * b, c["cached"], h, d))
    if kind == "layer":
        g = _generator(seed)
        b, s, h, d = c["batch"], c["tokens"], c["heads"], c["d"]
        nd = h * d
        qkv = _rows(g, b, s, 3 * nd)
        t = [qkv[..., :nd], qkv[..., nd:2 * nd], qkv[..., 2 * nd:], _rows(g, b, s, 3 * h), _rows(g, b, s, h),
             _rows(g, b * h, s, d), 1.0 + 0.1 * _rows(g, d, dtype=F32), _rows(g, b, s, nd), _rows(g, b, s, nd)]
        tables = lo.rotary_tables(c["rotary"], s, device="cuda") + (c["rotary"],) if c["rotary"] else None
        if not c["train"]:
            return dict(case=c, t=t, tables=tables)
        douts = [_rows(g, b * h, s, d) for _ in range(3)] + [_rows(g, b * h, s, 1, dtype=F32) for _ in range(4)] + [_rows(g, b, s, nd)]
        return dict(case=c, t=_leaves(t), tables=tables, douts=douts)
    raise ValueError(kind)


# ---------------------------------------------------------------------------------------------------------- one call
def _with_gradients(outs, douts, leaves):
    leaves = [t for t in leaves if t is not None]
    return [o.detach() for o in outs] + list(torch.autograd.grad(outs, leaves, douts))


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "causal":
        o = _CAUSAL[c["form"]](*state["args"], chunk_size=c["chunk"], use_muon=c["muon"], momentum=state["gate"])
        return _with_gradients([o], [state["dout"]], state["args"] + [state["gate"]]) if c["train"] else o
    if kind == "ffn":
        return lb.fused_swiglu_ffn_fwd(state["w02"], state["w1"], state["x"])
    if kind == "bidirectional":
        return lb.bidirectional_lact_swiglu(*state["args"], use_muon=c["muon"])
    if kind == "nvs":
        o, w0, w1, w2 = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*state["args"], state["order"],
                                                                              muon_update_steps=c["muon_steps"])
        return _with_gradients([o], [state["dout"]], state["args"]) if c["train"] else [o, w0, w1, w2]
    if kind == "video":
        o, w0, w1, w2 = lb.ar_fast_weight_swish_glu_weight_norm_mini_batch_with_momentum(
            *state["args"], 1.0, mini_batch_size=c["frame"], update_every=c["spacing"] * c["frame"], use_moun=c["muon"],
            num_moun_iters=5, fw_momentum=state["gate"], use_momentum=c["momentum"])
        return _with_gradients([o], [state["dout"]], state["args"] + [state["gate"]]) if c["train"] else [o, w0, w1, w2]
    if kind == "video_step":
        return lb.ar_fast_weight_swish_glu_weight_norm_mini_batch_inference_with_momentum(
            *state["args"], 1.0, mini_batch_size=c["frame"], do_update=c["update"], use_moun=c["muon"], num_moun_iters=5,
            fw_momentum=state["gate"], dw0_momentum=state["m"][0], dw1_momentum=state["m"][1], dw2_momentum=state["m"][2],
            use_momentum=True)
    if kind == "window":
        o = lo.sliding_window_attention(state["q"], state["k"], state["v"], c["window"], cu_seqlens=state["cu"])
        return _with_gradients([o], [state["dout"]], [state["q"], state["k"], state["v"]]) if c["train"] else o
    if kind == "cache":
        return lo.sliding_window_attention_inference(state["q"], state["k"], state["v"], c["tokens"], kv_cache=state["cache"])
    if kind == "layer":
        xq, xk, xv, lr, gate, fw_x, weight, scale, attn = state["t"]
        outs = list(lo.qkv_prologue(xq, xk, xv, c["heads"], rotary=state["tables"]))
        outs += list(lo.lr_prologue(lr, c["heads"], 0.01, gate))
        outs.append(lo.out_epilogue(fw_x, weight, c["heads"], scale, attn))
        return _with_gradients(outs, state["douts"], state["t"]) if c["train"] else outs
    raise ValueError(kind)


# ---------------------------------------------------------------------------------------------------------- bounds
def _newton_schulz_flops(r, c, steps):
    m, n = min(r, c), max(r, c)
    return steps * (4 * m * m * n + 2 * m ** 3)


def _recurrence_work(c, tokens, read, updated, updates, train, muon, concat=False, momentum=False, act=2, lr=4, state_out=False):
    """One pass of a recurrence over `units` entries: `read` tokens applied, `updated` tokens contracted in `updates`
    updates.  The backward has twice the products of the forward (Newton-Schulz included)."""
    b, d, h = c["units"], c["d"], c["h"]
    flops = 6 * d * h * read + 12 * d * h * updated
    if muon:
        ns = _newton_schulz_flops(2 * h, d, muon) if concat else 2 * _newton_schulz_flops(h, d, muon)
        flops += updates * (ns + _newton_schulz_flops(d, h, muon))
    weights = 3 * d * h * 4
    inputs = weights + 3 * d * tokens * act + 3 * tokens * lr + (4 * tokens if momentum else 0)
    out = read * d * act
    if train:   # every input read again for its gradient and the gradients written
        return dict(bytes=b * (2 * inputs + 2 * out + inputs), flops=3 * b * flops)
    return dict(bytes=b * (inputs + out + (weights if state_out else 0)), flops=b * flops)


def _window_pairs(n, window):
    """(query, key) pairs of a causal band over n tokens."""
    w = min(window, n)
    return w * (w + 1) // 2 + (n - w) * w


def work(case):
    c, kind = case, case["kind"]
    if kind == "causal":
        updates = len(range(0, c["tokens"] - c["chunk"], c["chunk"]))
        return _recurrence_work(c, c["tokens"], c["tokens"], updates * c["chunk"], updates, c["train"], 5 if c["muon"] else 0,
                                concat=c["form"].endswith("fused"), momentum=c["momentum"], lr=2 if c["lr"] == "bf16" else 4)
    if kind == "ffn":
        b, n, d, h = c["units"], c["tokens"], c["d"], c["h"]
        return dict(bytes=b * (3 * d * h + 2 * n * d) * 2, flops=6 * b * n * d * h)
    if kind == "bidirectional":
        n = c["tokens"]
        return _recurrence_work(c, n, n, n, 1, False, 5 if c["muon"] else 0, act=2 if c["dtype"] == "bf16" else 4)
    if kind == "nvs":
        n = c["inputs"] + c["targets"]
        w = _recurrence_work(c, n, n if c["all_tokens"] else c["targets"], c["inputs"], 1, c["train"], c["muon_steps"], state_out=True)
        if not c["all_tokens"]:   # queries of the input tokens, keys and values of the target tokens are never needed
            w["bytes"] -= c["units"] * c["d"] * 2 * (c["inputs"] + 2 * c["targets"]) * (3 if c["train"] else 1)
        return w
    if kind == "video":
        n = _video_length(c)
        return _recurrence_work(c, n, n, c["frames"] * c["frame"], c["frames"], c["train"], 5 if c["muon"] else 0,
                                momentum=c["momentum"], state_out=True)
    if kind == "video_step":
        n, u = c["frame"], c["update"]
        w = _recurrence_work(c, n, n, n if u else 0, 1 if u else 0, False, 5 if c["muon"] else 0, momentum=u, state_out=True)
        if u:      # momentum state in and out
            w["bytes"] += c["units"] * 2 * 3 * c["d"] * c["h"] * 4
        else:      # keys, values and learning rates are not needed
            w["bytes"] -= c["units"] * (2 * c["d"] * 2 + 3 * 4) * n
        return w
    if kind == "window":
        b, n, h, d, s = (c["batch"] if c["sequences"] == 1 else 1), c["tokens"], c["heads"], c["d"], c["sequences"]
        pairs = b * h * s * _window_pairs(n // s, c["window"])
        tensor = b * n * h * d * 2
        return dict(bytes=tensor * (8 if c["train"] else 4), flops=pairs * d * (4 + 10 if c["train"] else 4))
    if kind == "cache":
        b, n, h, d = c["batch"], c["tokens"], c["heads"], c["d"]
        return dict(bytes=b * h * d * 2 * (4 * n + 2 * c["cached"]), flops=4 * b * h * d * n * (n + c["cached"]))
    if kind == "layer":
        b, s, h, d = c["batch"], c["tokens"], c["heads"], c["d"]
        big, small = b * s * h * d * 2, b * s * h * (4 * 2 + 4 * 4)
        # forward: three projections in and out, then three tensors in and one out; backward: inputs and gradients in,
        # gradients out (the gradient of the attention output is the output's own)
        return dict(bytes=10 * big + small + (15 * big + 2 * small if c["train"] else 0),
                    flops=b * s * h * d * (40 + (80 if c["train"] else 0)))
    raise ValueError(kind)


def tolerance(case):
    c, kind = case, case["kind"]
    if kind in ("causal", "video", "video_step", "nvs", "bidirectional"):
        if c.get("muon", True) and c.get("muon_steps", 5) > 0 and c.get("update", True):
            # Newton-Schulz in bf16: one flipped rounding of the gradient moves its result by 1e-2, and the recurrence
            # carries that on
            return dict(rel=3e-2, max=0.99)
        if c.get("dtype") == "f32":
            return dict(rel=1e-5)
        # bf16 planes between the products, up to 16 sequential updates; gradients go through two such passes
        return dict(rel=2e-2, max=0.8)
    return dict(rel=1e-2)
