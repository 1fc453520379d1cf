"""Row-wise stages of the LaCT layer around the chunk recurrence (the layer's own code,
lact_llm/lact_model/layer_lact_swiglu.py, is outside this package; these are the passes over
[b, s, n_h * d] that sit directly on the recurrence's inputs and output).

Forward: one fused CUDA pass each.  Backward (training): one fused pass each that recomputes from the saved inputs (the
forward's bf16 roundings are treated as identities).  Registered operators, csrc/native/layer.cpp and attention.cpp.

Attention half of the hybrid layers (tcgen05 kernels, forward and backward, head dimension 64 or 128):
`sliding_window_attention` (causal band; packed sequences by `cu_seqlens`, padded batches by `attention_mask`),
`block_attention` (not causal, own key count) and, under the reference's names, the autoregressive-video layer's
`batched_sliding_window_attention`, `batched_sliding_window_attention_with_repeated_chunks` and
`sliding_window_attention_inference`."""
from __future__ import annotations

import math
from typing import Optional, Tuple

import torch

from . import _lib as L
from .ops import _op

BF16 = torch.bfloat16


def _seq_start(cu_seqlens: torch.Tensor, n_tokens: int, device) -> torch.Tensor:
    """int32 [n_tokens]: for every token of a packed batch entry, the first token of its sequence (no host
    synchronisation: the output size is known)."""
    if cu_seqlens.is_cuda and cu_seqlens.device == torch.device(device):
        return L.call(_op("seq_start"), cu_seqlens, n_tokens)
    cu = cu_seqlens.to(device=device, dtype=torch.int64)
    return torch.repeat_interleave(cu[:-1], cu[1:] - cu[:-1], output_size=n_tokens).to(torch.int32).contiguous()


def rotary_tables(head_dim: int, n_positions: int, base: float = 500000.0, device=None, dtype=BF16):
    """cos / sin tables [n_positions, head_dim / 2] as fla.modules.RotaryEmbedding(dim=head_dim, base=rope_theta)
    caches them (fp32 inverse frequencies and positions, result cast to the activations' dtype)."""
    inv_freq = 1.0 / (base ** (torch.arange(0, head_dim, 2, dtype=torch.float32, device=device) / head_dim))
    freqs = torch.outer(torch.arange(n_positions, dtype=torch.float32, device=device), inv_freq)
    return torch.cos(freqs).to(dtype), torch.sin(freqs).to(dtype)


def qkv_prologue(xq: torch.Tensor, xk: torch.Tensor, xv: torch.Tensor, num_heads: int, qkv_silu: bool = True,
                 no_v_silu: bool = False, rotary: Optional[Tuple[torch.Tensor, torch.Tensor, int]] = None,
                 seqlen_offset: int = 0, cu_seqlens: Optional[torch.Tensor] = None):
    """fast_q, fast_k, fast_v of layer_lact_swiglu.py:399-446 in one pass: `[b, s, (n_h d)] -> [(b n_h), s, d]`, SiLU
    on q, k (and v unless `no_v_silu`), per-head l2_norm of q and k (ttt_operation.py:19-26) and, when `rotary` =
    (cos, sin, attention_head_dim) is given (`ttt_nope` off), the rotary embedding of q and k over attention heads of
    that size (tables as `rotary_tables` / fla.modules.RotaryEmbedding build them, bf16 [positions, head_dim / 2]).
    Inputs may be views of a fused projection.  Differentiable (see the module docstring).  `cu_seqlens` (with
    `rotary`, batch of one): sequences packed back to back, positions restart at every sequence start (:434)."""
    if not (xq.is_cuda and xk.is_cuda and xv.is_cuda):
        raise ValueError("qkv_prologue needs CUDA tensors (there is no CPU implementation)")
    assert xq.shape == xk.shape == xv.shape and xq.dim() == 3 and xq.shape[2] % num_heads == 0
    assert xq.dtype == xk.dtype == xv.dtype == BF16, "expected [b, s, n_heads * d] bf16 tensors"
    cos = sin = None
    rope_hd = 0
    if rotary is not None:
        cos, sin, rope_hd = rotary
        assert cos.dtype == BF16 and sin.dtype == BF16 and cos.shape == sin.shape and cos.shape[1] * 2 == rope_hd
        cos, sin = cos.contiguous(), sin.contiguous()
    seq_start = None
    if cu_seqlens is not None and rotary is not None:
        if xq.shape[0] != 1:
            raise ValueError("packed sequences (cu_seqlens) need a batch of one")
        seq_start = _seq_start(cu_seqlens, xq.shape[1], xq.device)
    q, k, v = L.call(_op("qkv_prologue"), xq, xk, xv, num_heads, bool(qkv_silu), not no_v_silu, cos, sin, int(rope_hd),
                     int(seqlen_offset), seq_start)
    return q, k, v


def lr_prologue(lr_proj: torch.Tensor, num_heads: int, base_lr: float, momentum_logits: torch.Tensor = None):
    """fw_lr1, fw_lr2, fw_lr3 (and momentum) of layer_lact_swiglu.py:463-480: softplus(lr_proj.float() +
    inv_softplus(base_lr)) split per head into three fp32 [(b n_h), s, 1] tensors; `momentum_logits` is the output of
    the momentum Linear BEFORE its Sigmoid ([b, s, n_h]); the result is sigmoid(.) in the logits' dtype, as float.
    Differentiable with respect to the projections."""
    if not lr_proj.is_cuda:
        raise ValueError("lr_prologue needs CUDA tensors (there is no CPU implementation)")
    assert lr_proj.dim() == 3 and lr_proj.shape[2] == 3 * num_heads
    if momentum_logits is not None:
        assert momentum_logits.shape == (*lr_proj.shape[:2], num_heads)
    base_lr_inv = base_lr + math.log(-math.expm1(-base_lr))
    outs = L.call(_op("lr_prologue"), lr_proj, momentum_logits, num_heads, base_lr_inv)
    return outs[0], outs[1], outs[2], outs[3] if len(outs) == 4 else None


def out_epilogue(fw_x: torch.Tensor, norm_weight: torch.Tensor, num_heads: int, scale_proj: torch.Tensor = None,
                 o: torch.Tensor = None, eps: float = 1e-5) -> torch.Tensor:
    """`o + merge_heads(ttt_norm(fw_x) * silu(scale_proj))` of layer_lact_swiglu.py:556-568 in one pass.
    fw_x: [(b n_h), s, d] bf16 (output of the recurrence); norm_weight: [d]; scale_proj (the output of
    `ttt_scale_proj`, before its SiLU) and o (attention output): [b, s, n_h * d] bf16 or None.
    Differentiable with respect to fw_x, the norm weight, scale_proj and o."""
    if not fw_x.is_cuda:
        raise ValueError("out_epilogue needs CUDA tensors (there is no CPU implementation)")
    assert fw_x.dim() == 3 and fw_x.dtype == BF16 and fw_x.shape[0] % num_heads == 0
    B, s, d = fw_x.shape
    assert norm_weight.shape == (d,)
    for t, name in ((scale_proj, "scale_proj"), (o, "o")):
        assert t is None or (t.shape == (B // num_heads, s, num_heads * d) and t.dtype == BF16), \
            f"{name}: expected a [b, s, n_heads * d] bf16 tensor"
    return L.call(_op("out_epilogue"), fw_x, norm_weight, scale_proj, o, num_heads, float(eps))


# ------------------------------------------------------------------------------------------ sliding-window attention
def sliding_window_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, window_size: Optional[int] = None,
                             softmax_scale: Optional[float] = None,
                             cu_seqlens: Optional[torch.Tensor] = None,
                             attention_mask: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Causal attention over the last `window_size` keys (the query's own position included), q, k, v and the
    result [b, l, n_heads, head_dim] bf16: what `flash_attn_func(q, k, v, causal=True, window_size=(window_size - 1,
    0))` computes at lact_llm/lact_model/layer_lact_swiglu.py:386-394 and
    minimal_implementations/causal_lact_with_sliding_window_attn.py:380-384 (`window_size=None`: all earlier keys).
    head_dim 64 or 128.  Differentiable (dq, dk, dv by `lact_swa_bwd`).  `cu_seqlens` (int32 [n + 1], device): the batch
    entry (b must be 1) is n sequences packed back to back, as for `flash_attn_varlen_func` (:371-385): no query sees
    a key of an earlier sequence.  `attention_mask` ([b, l], nonzero = token, zero = padding, any padding side): the
    padded-batch branch (:351-370): the real tokens of all entries are gathered into one packed entry, attended per
    sequence and scattered back, padding positions of the result are zero (`unpad_input` / `pad_input`).  Like the
    reference's, this branch reads the number of real tokens on the host."""
    if not (q.is_cuda and k.is_cuda and v.is_cuda):
        raise ValueError("sliding_window_attention needs CUDA tensors (there is no CPU implementation)")
    assert q.dim() == 4 and q.shape == k.shape == v.shape, "q, k, v: [b, l, n_heads, head_dim], equal head counts"
    assert q.dtype == k.dtype == v.dtype == BF16, "bf16 activations"
    if q.shape[3] not in (64, 128):
        raise ValueError("head_dim must be 64 or 128")
    scale = float(softmax_scale) if softmax_scale is not None else q.shape[3] ** -0.5
    window = int(window_size) if window_size else 0
    if attention_mask is not None:
        if cu_seqlens is not None:
            raise ValueError("give attention_mask or cu_seqlens, not both")
        b, l, h, d = q.shape
        assert attention_mask.shape == (b, l), "attention_mask: [b, l]"
        mask = attention_mask.to(device=q.device) != 0
        idx = torch.nonzero(mask.reshape(-1)).reshape(-1)   # (host synchronisation: data-dependent size)
        if idx.numel() == 0:
            return torch.zeros_like(q)
        cu = torch.nn.functional.pad(torch.cumsum(mask.sum(dim=1), 0), (1, 0)).to(torch.int32)
        packed = [t.reshape(b * l, h, d).index_select(0, idx).unsqueeze(0) for t in (q, k, v)]
        o = L.call(_op("swa_fwd"), *packed, window, scale, _seq_start(cu, idx.numel(), q.device))[0]
        return torch.zeros(b * l, h, d, dtype=q.dtype, device=q.device).index_copy(0, idx, o[0]).reshape(b, l, h, d)
    seq_start = None
    if cu_seqlens is not None:
        if q.shape[0] != 1:
            raise ValueError("packed sequences (cu_seqlens) need a batch of one")
        seq_start = _seq_start(cu_seqlens, q.shape[1], q.device)
    return L.call(_op("swa_fwd"), q, k, v, window, scale, seq_start)[0]


def block_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor,
                    softmax_scale: Optional[float] = None) -> torch.Tensor:
    """Full (not causal) attention of every query of a batch entry over all keys of that entry: q [b, lq, h, d],
    k, v [b, lk, h, d] bf16, result [b, lq, h, d].  What `flash_attention(q, k, v, k_lens=<all keys>, window_size=(-1,
    -1))` computes for the frame blocks of the autoregressive-video layer
    (lact_ar_video/minVid/models/blocks/ar_lact_swa_repeat.py:313-318, 344-364).  The same tcgen05 kernels as
    `sliding_window_attention`, band and sequence masks off.  head_dim 64 or 128.  Differentiable."""
    if not (q.is_cuda and k.is_cuda and v.is_cuda):
        raise ValueError("block_attention needs CUDA tensors (there is no CPU implementation)")
    assert q.dim() == 4 and k.shape == v.shape and k.dim() == 4, "q [b, lq, h, d]; k, v [b, lk, h, d]"
    assert q.shape[0] == k.shape[0] and q.shape[2:] == k.shape[2:], "q and k, v differ in the token count only"
    assert q.dtype == k.dtype == v.dtype == BF16, "bf16 activations"
    if q.shape[3] not in (64, 128):
        raise ValueError("head_dim must be 64 or 128")
    if q.shape[1] == 0 or k.shape[1] == 0:
        return torch.zeros_like(q)
    scale = float(softmax_scale) if softmax_scale is not None else q.shape[3] ** -0.5
    return L.call(_op("swa_fwd"), q, k, v, -1, scale, None)[0]


def batched_sliding_window_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, mini_batch_size: int,
                                     update_every: int, num_chunks: int, kv_cache_size: int) -> torch.Tensor:
    """The block attention of the autoregressive-video layer, same name and arguments as
    ar_lact_swa_repeat.py:299-365.  q, k, v: [b, l, h, d] with l = update_every - mini_batch_size + update_every *
    (num_chunks - 1).  The first update_every - mini_batch_size tokens attend among themselves; every later block of
    update_every tokens is a clean part (the first mini_batch_size tokens, attending among themselves) followed by a
    noisy part that attends over the last kv_cache_size clean keys and the keys after them (mini_batch_size +
    kv_cache_size keys, as the reference's k_lens says)."""
    b, l = q.shape[:2]
    first, n_c, mb = update_every - mini_batch_size, num_chunks - 1, mini_batch_size
    assert l == first + update_every * n_c, "l = update_every - mini_batch_size + update_every * (num_chunks - 1)"
    assert 0 <= kv_cache_size <= mb
    parts = [block_attention(q[:, :first], k[:, :first], v[:, :first])] if first > 0 else []
    if n_c > 0:
        q_r, k_r, v_r = (t[:, first:].reshape(b * n_c, update_every, *t.shape[2:]) for t in (q, k, v))
        o_clean = block_attention(q_r[:, :mb], k_r[:, :mb], v_r[:, :mb])
        k_end = min(update_every, 2 * mb)   # keys [mb - kv_cache_size, mb - kv_cache_size + (mb + kv_cache_size))
        o_noise = block_attention(q_r[:, mb:], k_r[:, mb - kv_cache_size:k_end], v_r[:, mb - kv_cache_size:k_end])
        parts.append(torch.cat([o_clean, o_noise], dim=1).reshape(b, n_c * update_every, *q.shape[2:]))
    return torch.cat(parts, dim=1) if len(parts) > 1 else parts[0]


def batched_sliding_window_attention_with_repeated_chunks(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor,
                                                          mini_batch_size: int, update_every: int, num_chunks: int,
                                                          kv_cache_size: int) -> torch.Tensor:
    """ar_lact_swa_repeat.py:368-463, same name and arguments: update_every = (num_repeat + 1) * mini_batch_size.  The
    first update_every - mini_batch_size tokens are num_repeat blocks of mini_batch_size tokens, each attending within
    itself; every later block of update_every tokens is a clean part (mini_batch_size tokens, attending within itself)
    and num_repeat noisy parts, each attending over the last kv_cache_size clean keys and its own keys."""
    b, l = q.shape[:2]
    first, n_c, mb = update_every - mini_batch_size, num_chunks - 1, mini_batch_size
    nr = update_every // mb - 1
    assert update_every == (nr + 1) * mb and nr >= 1, "update_every must be a multiple (>= 2) of mini_batch_size"
    assert l == first + update_every * n_c and 0 <= kv_cache_size <= mb
    tail = q.shape[2:]
    blocks = lambda t: t[:, :first].reshape(b * nr, mb, *tail)
    parts = [block_attention(blocks(q), blocks(k), blocks(v)).reshape(b, first, *tail)]
    if n_c > 0:
        q_r, k_r, v_r = (t[:, first:].reshape(b * n_c, update_every, *tail) for t in (q, k, v))
        o_clean = block_attention(q_r[:, :mb], k_r[:, :mb], v_r[:, :mb])
        noisy = lambda t: t[:, mb:].reshape(b * n_c * nr, mb, *tail)
        cached = lambda t: t[:, mb - kv_cache_size:mb].repeat_interleave(nr, dim=0)
        o_noise = block_attention(noisy(q_r), torch.cat([cached(k_r), noisy(k_r)], dim=1),
                                  torch.cat([cached(v_r), noisy(v_r)], dim=1)).reshape(b * n_c, nr * mb, *tail)
        parts.append(torch.cat([o_clean, o_noise], dim=1).reshape(b, n_c * update_every, *tail))
    return torch.cat(parts, dim=1) if len(parts) > 1 else parts[0]


def sliding_window_attention_inference(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, mini_batch_size: int,
                                       kv_cache: Optional[torch.Tensor] = None, interleave: bool = False,
                                       kv_cache_size: int = 1560) -> torch.Tensor:
    """ar_lact_swa_repeat.py:464-531, same name and arguments: the attention of one generation step of the
    autoregressive-video layer.  (1) no cache, not interleaved: full attention; (2) interleaved: the first
    mini_batch_size (clean) tokens attend among themselves, the rest over the last kv_cache_size clean keys and their
    own; (3) with a cache ([2 b, l_c, h, d]: keys of all entries, then values): full attention over cache + k."""
    if kv_cache is None and not interleave:
        return block_attention(q, k, v)
    if interleave:
        mb = mini_batch_size
        o_clean = block_attention(q[:, :mb], k[:, :mb], v[:, :mb])
        o_rest = block_attention(q[:, mb:], k[:, mb - kv_cache_size:], v[:, mb - kv_cache_size:])
        return torch.cat([o_clean, o_rest], dim=1)
    k_cache, v_cache = kv_cache.chunk(2, dim=0)
    every = (q, k_cache, v_cache, k, v)
    if (all(t.is_cuda and t.dtype == BF16 and t.dim() == 4 and t.device == q.device for t in every) and k.shape == v.shape
            and k_cache.shape == v_cache.shape and all(t.shape[0] == q.shape[0] and t.shape[2:] == q.shape[2:] for t in every)
            and q.shape[3] in (64, 128) and min(t.shape[1] for t in every) > 0):
        return L.call(_op("swa_fwd_cache"), *every, q.shape[3] ** -0.5)   # (the keys are read where they lie)
    return block_attention(q, torch.cat([k_cache, k], dim=1), torch.cat([v_cache, v], dim=1))
