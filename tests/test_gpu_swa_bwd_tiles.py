"""Attention backward at the edges of its 128-row tiles: gradients against fp64 autograd."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (entries, queries, keys, heads, d, window; window < 0: block attention): one, two, three and more inner tiles on either side,
# lengths that end on, before and after a tile's edge, windows of a single key, of a tile and around it, wider than the sequence
@pytest.mark.parametrize("b,l,lk,h,d,window", [(1, 1, 1, 1, 128, 0), (2, 127, 127, 2, 64, 1), (1, 128, 128, 3, 128, 0),
                                               (1, 129, 129, 2, 128, 128), (2, 257, 257, 1, 64, 129), (1, 384, 384, 2, 128, 127),
                                               (1, 641, 641, 2, 128, 255), (1, 900, 900, 1, 64, 2000), (1, 1, 300, 2, 128, -1),
                                               (2, 130, 127, 2, 64, -1), (1, 256, 513, 1, 128, -1), (1, 500, 1, 2, 128, -1)])
def test_gradients(b, l, lk, h, d, window):
    _check(b, l, lk, h, d, window)


# sequences packed back to back: many in a tile and one over many, ends on, before and after the edges of tiles and of the 32 rows
# of a warp, windows shorter and longer than a sequence
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [0, 1, 40, 128, 700])
@pytest.mark.parametrize("lengths", [(1, 30, 1, 2, 94, 128, 129, 127, 300), (640,), (5,) * 70, (1000, 3, 29, 1, 31), (257, 511)])
def test_gradients_of_packed_sequences(d, window, lengths):
    _check(1, sum(lengths), sum(lengths), 2, d, window, lengths)


def _check(b, l, lk, h, d, window, lengths=None):
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(l * 7 + lk)
    rn = lambda n: torch.randn(b, n, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v, do = rn(l), rn(lk), rn(lk), rn(l)
    ref = [t.double().transpose(1, 2).requires_grad_(True) for t in (q, k, v)]
    s, start = ref[0] @ ref[1].transpose(2, 3) * d ** -0.5, None
    if window >= 0:
        i, j = torch.arange(l, device="cuda")[:, None], torch.arange(lk, device="cuda")[None]
        if lengths is not None:
            start = torch.cat([torch.full((n,), sum(lengths[:m]), device="cuda") for m, n in enumerate(lengths)]).int()
            s = s.masked_fill(j < start[:, None], float("-inf"))
        s = s.masked_fill((j > i) | ((j <= i - window) if window > 0 else torch.zeros_like(j > i)), float("-inf"))
    out = s.softmax(-1) @ ref[2]
    want = [t.transpose(1, 2) for t in torch.autograd.grad(out, ref, do.double().transpose(1, 2))]
    o = out.transpose(1, 2).to(torch.bfloat16).reshape(-1).view(b, l, h, d)
    lse = (s.logsumexp(-1) * 1.4426950408889634).float().contiguous()
    dq, dk, dv = (torch.full_like(t, float("nan")) for t in (q, k, v))
    delta = torch.empty(b, h, l, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    st = lambda t: (h * d, t.shape[1] * h * d)   # contiguous (strides of length-one axes are anything)
    L.check(L.lib().lact_swa_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(), dq.data_ptr(),
                                 dk.data_ptr(), dv.data_ptr(), delta.data_ptr(), b, l, lk, h, d, *st(q), *st(k), *st(v), *st(o), *st(do),
                                 window, d ** -0.5, start.data_ptr() if lengths is not None else None, status.data_ptr(), L.stream_ptr()), "bwd")
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    for got, w, like in zip((dq, dk, dv), want, (q, k, v)):
        # P and dS are rounded to bf16 (2^-9), so are the results; dS = P (dP - delta) cancels, at worst wholly (one visible key):
        # what is left is compared on the scale of the terms, |dP| ~ sqrt(d) times the other operand
        scale = max(float(w.norm()), 2.0 ** -2 * float(like.double().norm()))
        assert bool(torch.isfinite(got).all()) and float((got.double() - w).norm()) <= 1e-2 * scale
