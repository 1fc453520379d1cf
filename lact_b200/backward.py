"""Newton-Schulz with kept iterates and its backward, and the strided product entry, called one by one from Python: what the
stand-alone `zeropower_via_newtonschulz5` differentiates with.  (The recurrence's own backward is the registered operator
`lact_b200::scan_bwd`, csrc/native/scan_bwd.cpp.)"""
from __future__ import annotations

import ctypes as C
from typing import Dict

import torch

from . import _lib as L

BF16 = torch.bfloat16
_status: Dict[tuple, torch.Tensor] = {}


def _status_word(dev: torch.device) -> torch.Tensor:
    """Device status word of the backward kernels, one per (device, stream)."""
    key = (dev.index if dev.index is not None else torch.cuda.current_device(), L.stream_ptr())
    if key not in _status:
        L.prepare_status(dev)
        _status[key] = torch.zeros(64, dtype=torch.int32, device=dev)
    return _status[key]


def reset_status(dev: torch.device) -> None:
    """Clears the word (stream-ordered): kernels return early while it is non-zero, so a call must not inherit the failure
    of an earlier one (which stays on record for the host, see `_lib.mark_pending`)."""
    _status_word(dev).zero_()


def post_status(dev: torch.device) -> None:
    """After the kernels have been enqueued: raises if an earlier call has recorded a failure by now."""
    L.mark_pending(_status_word(dev).view(torch.uint8))


def check_status(dev: torch.device) -> None:
    """Raises if a bounded wait ran out during the sweep; the word is cleared first, so the next
    backward call starts clean."""
    word = _status_word(dev)
    st = int(word[0].item())
    if st != 0:
        word.zero_()
        raise L.LactError(f"device status {st} during backward")


def _strided(t):
    """A [batch, rows, cols] bf16 tensor as (tensor, row stride, batch stride) for the strided GEMM entry; views
    whose innermost axis is contiguous and whose strides / base keep 16-byte alignment pass through uncopied."""
    if t.stride(2) != 1 or t.stride(1) % 8 or t.stride(0) % 8 or t.data_ptr() % 16 or t.stride(1) < t.shape[2]:
        t = t.contiguous()
    return t, t.stride(1), t.stride(0)


def _desc(a, b, a_mn=False, b_mn=False, a1=None, b1=None, a1_mn=False, b1_mn=False, out=None,
          out_dtype=torch.float32, accumulate=False):
    """(lact_bmm_desc, output tensor, tensors to keep alive) for c[batch, M, N] (+)= a b^T (+ a1 b1^T)."""
    a, a_ld, a_bs = _strided(a)
    b, b_ld, b_bs = _strided(b)
    batch = a.shape[0]
    M, K = (a.shape[2], a.shape[1]) if a_mn else (a.shape[1], a.shape[2])
    N = b.shape[2] if b_mn else b.shape[1]
    if out is None:
        out = torch.empty(batch, M, N, dtype=out_dtype, device=a.device)
    assert out.stride(2) == 1 and out.shape == (batch, M, N)
    a1_ld = a1_bs = b1_ld = b1_bs = 0
    if a1 is not None:
        a1, a1_ld, a1_bs = _strided(a1)
        b1, b1_ld, b1_bs = _strided(b1)
    d = L.BmmDesc(a.data_ptr(), b.data_ptr(), a1.data_ptr() if a1 is not None else None,
                  b1.data_ptr() if b1 is not None else None, out.data_ptr(), a_ld, a_bs, b_ld, b_bs, a1_ld, a1_bs,
                  b1_ld, b1_bs, out.stride(1), out.stride(0), batch, M, N, K, int(a_mn), int(b_mn), int(a1_mn),
                  int(b1_mn), L.dtype_code(out), int(accumulate))
    return d, out, (a, b, a1, b1)


def gemm(a, b, **kw):
    """c[batch, M, N] (+)= a b^T (+ a1 b1^T).  Operands bf16, [batch, rows, K] or (``*_mn``) [batch, K, rows];
    operands and `out` may be views into larger tensors (token ranges).  Keywords: a_mn, b_mn, a1, b1, a1_mn, b1_mn,
    out, out_dtype (fp32), accumulate."""
    reset_status(a.device)
    d, out, _keep = _desc(a, b, **kw)
    rc = L.lib().lact_bmm_group_bf16(C.byref(d), 1, _status_word(out.device).data_ptr(), L.stream_ptr())
    L.check(rc, "lact_bmm_group_bf16")
    return out


def ns_forward_saved(G, steps, const_coeffs, gram_right):
    """Recomputes the Newton-Schulz iteration on G [nmat, R, C] keeping every iterate
    (`lact_ns_trace_fwd`: the forward kernels' own arithmetic, iterates in a trace buffer).
    Returns a dict used by `ns_backward` and the result U in G's orientation (bf16)."""
    G = G.contiguous()
    nmat, R, Cc = G.shape
    if G.dtype not in (torch.float32, BF16):
        G = G.float()
    G = L.on_16_bytes(G)
    if int(steps) == 0:   # no iteration (lact_nvs/lact_ttt.py with muon_update_steps = 0): the normalisation alone
        from . import ops
        U = ops.zeropower_via_newtonschulz5(G, 0)
        return dict(trace=None, shape=(nmat, R, Cc), steps=0, cc=1, gr=int(bool(gram_right)), G=G), U
    reset_status(G.device)
    need = C.c_size_t(0)
    L.check(L.lib().lact_ns_trace_bytes(nmat, R, Cc, int(steps), C.byref(need)), "lact_ns_trace_bytes")
    trace = torch.empty(need.value, dtype=torch.uint8, device=G.device)
    U = torch.empty(nmat, R, Cc, dtype=BF16, device=G.device)
    with torch.cuda.device(G.device):
        L.check(L.lib().lact_ns_trace_fwd(G.data_ptr(), L.dtype_code(G), U.data_ptr(), nmat, R, Cc, int(steps),
                                          int(bool(const_coeffs)), int(bool(gram_right)), trace.data_ptr(), trace.numel(),
                                          _status_word(G.device).data_ptr(), L.stream_ptr()), "lact_ns_trace_fwd")
    return dict(trace=trace, shape=(nmat, R, Cc), steps=int(steps), cc=int(bool(const_coeffs)), gr=int(bool(gram_right)),
                G=G), U


def ns_backward(saved, dU):
    """Gradient w.r.t. G of U = NS(G) given dU (fp32, G's orientation): `lact_ns_trace_bwd` walks
    the saved iterates backwards (three two-product contractions per iteration, roundings treated
    as identities, bf16 operands as in the reference's autograd), then the Frobenius
    normalisation X0 = bf16(G) / (||G|| + 1e-7) is differentiated here."""
    nmat, R, Cc = saved["shape"]
    reset_status(dU.device)
    du = (dU if dU.dtype == BF16 else dU.to(BF16)).contiguous()
    dX0 = torch.empty(nmat, R, Cc, dtype=torch.float32, device=du.device)
    trace = saved["trace"]
    if saved["steps"] == 0:
        dX0.copy_(du)
    with torch.cuda.device(du.device):
        if saved["steps"] > 0:
            L.check(L.lib().lact_ns_trace_bwd(du.data_ptr(), dX0.data_ptr(), nmat, R, Cc, saved["steps"], saved["cc"],
                                              saved["gr"], trace.data_ptr(), trace.numel(),
                                              _status_word(du.device).data_ptr(), L.stream_ptr()), "lact_ns_trace_bwd")
    # dX0 / den - bf16(G) <dX0, bf16(G)> / (den^2 ||bf16(G)||), in place in dX0
    G = saved["G"]
    G = G if (G.dtype == torch.float32 and G.is_contiguous()) else G.float().contiguous()
    part = torch.empty(nmat * 2 * L.lib().lact_momentum_bwd_slices(), dtype=torch.float32, device=du.device)
    L.check(L.lib().lact_ns_norm_bwd(G.data_ptr(), dX0.data_ptr(), part.data_ptr(), nmat, R * Cc, L.stream_ptr()),
            "lact_ns_norm_bwd")
    return dX0


def ns_backward_groups(saved, dUs):
    """`ns_backward` for one or two groups of matrices at once: all iterations of all groups in one cooperative
    launch (`lact_ns_trace_bwd_fused`) when an instantiation covers the shapes, else one group after the other."""
    same = all(sv["steps"] == saved[0]["steps"] and sv["cc"] == saved[0]["cc"] and sv["gr"] == saved[0]["gr"]
               for sv in saved)
    if same and 1 <= saved[0]["steps"] <= 5 and len(saved) <= 2:
        dev = dUs[0].device
        reset_status(dev)
        slices = L.lib().lact_momentum_bwd_slices()
        groups = (L.NsBwdGroup * len(saved))()
        keep, outs = [], []
        for i, (sv, dU) in enumerate(zip(saved, dUs)):
            nmat, R, Cc = sv["shape"]
            du = (dU if dU.dtype == BF16 else dU.to(BF16)).contiguous()
            G = sv["G"]
            G = G if (G.dtype == torch.float32 and G.is_contiguous()) else G.float().contiguous()
            dg = torch.empty(nmat, R, Cc, dtype=torch.float32, device=dev)
            part = torch.empty(nmat * 2 * slices, dtype=torch.float32, device=dev)
            keep += [du, G, part]
            outs.append(dg)
            groups[i] = L.NsBwdGroup(du.data_ptr(), G.data_ptr(), dg.data_ptr(), sv["trace"].data_ptr(),
                                     sv["trace"].numel(), part.data_ptr(), nmat, R, Cc)
        with torch.cuda.device(dev):
            rc = L.lib().lact_ns_trace_bwd_fused(groups, len(saved), saved[0]["steps"], saved[0]["cc"], saved[0]["gr"],
                                                 _status_word(dev).data_ptr(), L.stream_ptr())
        if rc == 0:
            return outs
        if rc != L.ERR_CONFIG:
            L.check(rc, "lact_ns_trace_bwd_fused")
    return [ns_backward(sv, dU) for sv, dU in zip(saved, dUs)]
