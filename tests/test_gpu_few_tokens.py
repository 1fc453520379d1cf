"""Apply on a few tokens by one cluster per entry: the bits of the two launches that more tokens take."""
import ctypes as C

import pytest
import torch

import lact_b200 as lb

pytestmark = pytest.mark.gpu


def _weights(b, d, h, g):
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    return rn(b, 2 * h, d) / d ** 0.5, rn(b, d, h) / h ** 0.5


# clusters of one to eight CTAs, fewer output features than hidden ones (48 per CTA at 192 of 256: a warp's last lanes have none), token counts around the steps of 16, and the largest that
# fit; more entries than clusters that run at once take two launches either way
@pytest.mark.parametrize("b,d,h", [(1, 64, 64), (3, 192, 192), (4, 384, 384), (2, 512, 512), (2, 128, 256), (2, 64, 448), (40, 256, 256), (2, 192, 256)])
@pytest.mark.parametrize("n", [1, 15, 17, 48, 64])
def test_same_bits_as_two_launches(b, d, h, n):
    g = torch.Generator(device="cuda").manual_seed(n + d)
    w02, w1 = (w.bfloat16() for w in _weights(b, d, h, g))
    x = torch.randn(b, 80, d, device="cuda", generator=g).bfloat16()
    want = lb.fused_swiglu_ffn_fwd(w02, w1, x)[:, :n]
    got = lb.fused_swiglu_ffn_fwd(w02, w1, x[:, :n].contiguous())
    assert torch.equal(got, want)


def test_views_and_neighbours():
    """A short range of a fused projection in the recurrence: strided tokens, nothing written beside the range."""
    g = torch.Generator(device="cuda").manual_seed(1)
    b, n, d, h = 2, 200, 128, 192
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    w = [rn(b, d, h) / d ** 0.5, rn(b, h, d) / h ** 0.5, rn(b, d, h) / d ** 0.5]
    qkv = rn(b, n, 3 * d).bfloat16()
    lr = [torch.rand(b, n, 1, device="cuda", generator=g) for _ in range(3)]
    q, k, v = (qkv[..., i * d:(i + 1) * d] for i in range(3))
    op = lb.TTTOperator
    run = lambda order: lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*w, q, k, v, *lr, order, muon_update_steps=0)[0]
    whole = run([op(0, n, False, True)])
    parts = run([op(0, 7, False, True), op(7, 190, False, True), op(190, n, False, True)])
    assert torch.equal(parts, whole)


@pytest.mark.parametrize("n", [5, 65])
@pytest.mark.parametrize("which", ["x", "out"])
def test_rows_off_16_bytes_are_refused(n, which):
    """As with more tokens, before any launch."""
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(3)
    w02, w1 = (w.bfloat16() for w in _weights(2, 64, 64, g))
    buf = {k: torch.zeros(2 * n * 64 + 8, dtype=torch.bfloat16, device="cuda") for k in ("x", "out")}
    hidden, word = torch.empty(2 * n * 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(64, dtype=torch.int32, device="cuda")
    p = lambda t, off=0: C.c_void_p(t.data_ptr() + off)
    call = lambda off: L.lib().lact_swiglu_ffn_apply(p(w02), p(w1), p(buf["x"], off if which == "x" else 0),
                                                     p(buf["out"], off if which == "out" else 0), p(hidden),
                                                     *map(C.c_int64, (2, n, 64, 64)), p(word), C.c_void_p(L.stream_ptr()))
    assert call(0) == 0
    torch.cuda.synchronize()
    assert call(2) == -2 and call(8) == -2


def test_nothing_is_written_after_an_earlier_failure():
    """(A status word that is set: the kernel stands aside, and so do all CTAs of a cluster.)"""
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(2)
    w02, w1 = (w.bfloat16() for w in _weights(2, 128, 128, g))
    x = torch.randn(2, 5, 128, device="cuda", generator=g).bfloat16()
    out, word = torch.full_like(x, 7), torch.full((64,), 101, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    rc = L.lib().lact_swiglu_ffn_apply(p(w02), p(w1), p(x), p(out), None, *map(C.c_int64, (2, 5, 128, 128)), p(word),
                                       C.c_void_p(L.stream_ptr()))
    assert rc == 0
    torch.cuda.synchronize()
    assert (out == 7).all()
