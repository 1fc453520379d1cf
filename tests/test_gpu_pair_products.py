"""Token x weight products on pairs of SMs: the same bits as the one-SM kernel gives entry by entry, and the fp32 reference."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# (entries, d, h, tokens, products that go to pairs): enough tiles of 256 tokens for the pairs in the batch and too few in a single
# entry.  Token counts at the edges of a tile and of either CTA's half of it, heads whose columns end inside a tile or whose k ends
# inside a k-block, the longest k that is kept in shared memory, two batch entries per pair and several, a tile for every entry
CASES = [(17, 384, 384, 3329, "gate down pointwise"), (46, 384, 384, 1153, "gate down pointwise"), (152, 192, 192, 1024, "gate down pointwise"),
         (90, 192, 192, 1409, "gate down pointwise"), (52, 256, 256, 2048 + 127, "gate down pointwise"), (64, 128, 256, 1560, "gate down pointwise"),
         (40, 512, 512, 1281, "gate down"), (60, 144, 80, 2560, "gate down pointwise"), (100, 64, 64, 2280, "gate pointwise"),
         (36, 320, 208, 1152 + 255, "gate pointwise"), (230, 384, 384, 250, "gate down pointwise")]
# calls that leave half of the second SM idle, load weights for every tile, or have column tiles that too few teams of pairs fit
SINGLE = [(300, 384, 384, 16, ""), (300, 384, 384, 128, ""), (300, 192, 192, 384, ""), (90, 512, 512, 16, ""), (40, 128, 256, 384, ""),
          (15, 384, 1600, 1024, ""), (9, 384, 2560, 1024, ""), (18, 512, 512, 4096, "gate down")]


def _on_pairs(call):
    """The products of a call that ran on pairs of SMs."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if "gemm_kernel" in e.name]
    assert names
    which = {"OpSwigluGate": "gate", "OpBmmStore": "down", "OpFwGradPointwise": "pointwise"}
    return {which[k] for k in which for n in names if k in n and "pair_gemm" in n}


def _inputs(b, d, h, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    w02, w1 = (rn(b, 2 * h, d) / d ** 0.5).bfloat16(), (rn(b, d, h) / h ** 0.5).bfloat16()
    kv = rn(b, n, 3 * d).bfloat16()   # k and v are views of a fused projection
    return w02, w1, kv[..., :d], kv[..., d:2 * d], [F.softplus(rn(b, n) - 2) for _ in range(3)]


def _close(got, want):
    # one rounding to bf16 (2^-9 relative) of fp32 sums, and of the hidden plane before the down projection
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -7


@pytest.mark.parametrize("b,d,h,n,pairs", CASES)
def test_apply(b, d, h, n, pairs):
    import lact_b200 as lb
    w02, w1, k, _, _ = _inputs(b, d, h, n, n)
    x = k.contiguous()
    out = lb.fused_swiglu_ffn_fwd(w02, w1, x)
    assert _on_pairs(lambda: lb.fused_swiglu_ffn_fwd(w02, w1, x)) == set(pairs.split()) - {"pointwise"}
    assert _on_pairs(lambda: lb.fused_swiglu_ffn_fwd(w02[:1], w1[:1], x[:1])) == set()
    for i in range(0, b, max(1, b // 4)):
        assert torch.equal(out[i], lb.fused_swiglu_ffn_fwd(w02[i:i + 1], w1[i:i + 1], x[i:i + 1])[0])
    y = x[-1].double() @ w02[-1].double().T
    _close(out[-1], (F.silu(y[:, :h]) * y[:, h:]) @ w1[-1].double().T)
    lb.synchronize_and_check()


@pytest.mark.parametrize("b,d,h,n,pairs", [c for c in CASES if "pointwise" in c[4]])
@pytest.mark.parametrize("lr_dtype", [torch.float32, torch.bfloat16, None])
def test_pointwise(b, d, h, n, pairs, lr_dtype):
    from lact_b200 import _lib as L
    w02, w1, k, v, lr = _inputs(b, d, h, n, n + 1)
    lr = [None] * 3 if lr_dtype is None else [t.to(lr_dtype) for t in lr]
    status = torch.zeros(64, dtype=torch.int32, device="cuda")

    def run(s):
        m = w02[s].shape[0]
        guard = torch.full((m * n * 3 * h + 2 * h,), -7.0, dtype=torch.bfloat16, device="cuda")
        dy, hid = guard[:m * n * 2 * h].view(m, n, 2 * h), guard[m * n * 2 * h:m * n * 3 * h].view(m, n, h)
        ptr = [t[s].data_ptr() if t is not None else None for t in lr]
        L.check(L.lib().lact_fw_grad_pointwise(w02[s].data_ptr(), w1[s].data_ptr(), k[s].data_ptr(), 3 * d, 3 * d * n, v[s].data_ptr(),
                                               3 * d, 3 * d * n, *ptr, 1 if lr_dtype == torch.bfloat16 else 0, n, 0.5, dy.data_ptr(),
                                               hid.data_ptr(), m, n, d, h, status.data_ptr(), L.stream_ptr()), "pointwise")
        assert bool((guard[m * n * 3 * h:] == -7).all())   # nothing is written behind the planes
        return dy, hid

    dy, hid = run(slice(0, b))
    assert _on_pairs(lambda: run(slice(0, b))) == {"pointwise"} and _on_pairs(lambda: run(slice(0, 1))) == set()
    for i in range(0, b, max(1, b // 4)):
        for got, want in zip((dy, hid), run(slice(i, i + 1))):
            assert torch.equal(got[i], want[0])
    kd, vd, l = k[-1].double(), v[-1].double(), [1.0 if t is None else t[-1].double()[:, None] for t in lr]
    y, dh = kd @ w02[-1].double().T, vd @ w1[-1].double()
    y0, y2, sg = y[:, :h], y[:, h:], torch.sigmoid(y[:, :h])
    _close(dy[-1][:, :h], 0.5 * l[0] * dh * y2 * sg * (1 + y0 * (1 - sg)))
    _close(dy[-1][:, h:], 0.5 * l[2] * dh * y0 * sg)
    _close(hid[-1], 0.5 * l[1] * y0 * sg * y2)
    assert int(status[0]) == 0


@pytest.mark.parametrize("b,d,h,n,pairs", SINGLE)
def test_calls_that_pairs_would_slow_down(b, d, h, n, pairs):
    import lact_b200 as lb
    w02, w1, k, v, lr = _inputs(b, d, h, n, n + 2)
    k, v = k.contiguous(), v.contiguous()
    assert _on_pairs(lambda: lb.fused_swiglu_ffn_fwd(w02, w1, k)) == set(pairs.split())
    assert _on_pairs(lambda: lb.fused_lact_swiglu_ffn_fast_weight_grads(w02, w1, k, v, *lr)) == set()
    lb.synchronize_and_check()


def _products(w02, w1, k, v, lr, status):
    """Apply and the pointwise stage through the C interface with a status word; the outputs, filled with -7 before."""
    from lact_b200 import _lib as L
    b, n, d = k.shape
    h = w1.shape[2]
    out, hidden, hid = (torch.full((b, n, w), -7.0, dtype=torch.bfloat16, device="cuda") for w in (d, h, h))
    dy = torch.full((b, n, 2 * h), -7.0, dtype=torch.bfloat16, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    L.check(L.lib().lact_swiglu_ffn_apply(ptr(w02), ptr(w1), ptr(k), ptr(out), ptr(hidden), *map(C.c_int64, (b, n, d, h)), ptr(status),
                                          C.c_void_p(L.stream_ptr())), "apply")
    L.check(L.lib().lact_fw_grad_pointwise(w02.data_ptr(), w1.data_ptr(), k.data_ptr(), d, d * n, v.data_ptr(), d, d * n,
                                           *[t.data_ptr() for t in lr], 0, n, 0.5, dy.data_ptr(), hid.data_ptr(), b, n, d, h,
                                           status.data_ptr(), L.stream_ptr()), "pointwise")
    torch.cuda.synchronize()
    return out, hidden, dy, hid


def test_after_an_earlier_failure_nothing_is_written():
    w02, w1, k, v, lr = _inputs(46, 384, 384, 1153, 3)
    k, v = k.contiguous(), v.contiguous()
    word = lambda x: torch.full((64,), x, dtype=torch.int32, device="cuda")
    assert _on_pairs(lambda: _products(w02, w1, k, v, lr, word(0))) == {"gate", "down", "pointwise"}
    status = word(101)
    assert all(bool((t == -7).all()) for t in _products(w02, w1, k, v, lr, status)) and int(status[0]) == 101


@pytest.mark.parametrize("b,d,h,n,_", SINGLE)
def test_a_pointwise_stage_that_pairs_would_slow_down(b, d, h, n, _):
    """The stage by itself: a gradient of heads of 128 features may run as one launch without it."""
    from lact_b200 import _lib as L
    w02, w1, k, v, lr = _inputs(b, d, h, n, n + 2)
    dy, hid, status = torch.empty(b, n, 2 * h, device="cuda").bfloat16(), torch.empty(b, n, h, device="cuda").bfloat16(), torch.zeros(64, dtype=torch.int32, device="cuda")
    call = lambda: L.check(L.lib().lact_fw_grad_pointwise(w02.data_ptr(), w1.data_ptr(), k.data_ptr(), 3 * d, 3 * d * n, v.data_ptr(), 3 * d, 3 * d * n,
                                                          *[t.data_ptr() for t in lr], 0, n, 0.5, dy.data_ptr(), hid.data_ptr(), b, n, d, h,
                                                          status.data_ptr(), L.stream_ptr()), "pointwise")
    assert _on_pairs(call) == set() and int(status[0]) == 0
