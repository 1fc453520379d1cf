"""fp32 mode: contractions in bf16 pieces at the edges of their tiles and slabs, and values that are no ordinary numbers."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lb():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lact_b200 import build
    build.build()
    import lact_b200
    return lact_b200


def _inputs(b, n, d, h, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = F.normalize(rn(b, n, d), dim=-1), F.normalize(rn(b, n, d), dim=-1)
    return [rn(b, h, d) / d ** 0.5, rn(b, d, h) / h ** 0.5, rn(b, h, d) / d ** 0.5, q, k, rn(b, n, d)] + \
        [F.softplus(rn(b, n, 1) - 2) for _ in range(3)]


def _gradients(w0, w1, w2, q, k, v, l0, l1, l2):
    y0, y2, dh = k @ w0.mT, k @ w2.mT, v @ w1
    s = torch.sigmoid(y0)
    return [(dh * y2 * s * (1 + y0 * (1 - s)) * l0).mT @ k, (v * l1).mT @ (y0 * s * y2), (dh * y0 * s * l2).mT @ k]


def _exact(w0, w1, w2, q, k, v, l0, l1, l2):
    """One update on all tokens, then apply, in 64 bits."""
    w0, w1, w2, q, k, v, l0, l1, l2 = (t.double() for t in (w0, w1, w2, q, k, v, l0, l1, l2))
    u = []
    for w, dw in zip((w0, w1, w2), _gradients(w0, w1, w2, q, k, v, l0, l1, l2)):
        x = w + dw
        u.append(x / (x.norm(dim=2, keepdim=True) + 1e-5) * w.norm(dim=2, keepdim=True))
    return (F.silu(q @ u[0].mT) * (q @ u[2].mT)) @ u[1].mT


# tokens around slabs of 64 and rows of 128; sides that 8, 64 and 128 do not divide; contractions cut into many and into one; rows past
# the end of a tile in a warp that has another tile to do (more entries than SMs)
@pytest.mark.parametrize("b,n,d,h", [(1, 1, 64, 64), (2, 63, 12, 8), (1, 65, 68, 72), (3, 129, 128, 128), (2, 1000, 100, 200),
                                     (1, 4100, 192, 192), (40, 200, 64, 128), (2, 300, 320, 136), (400, 33, 64, 72)])
def test_close_to_64_bits(lb, b, n, d, h):
    args = _inputs(b, n, d, h, seed=n)
    o = lb.bidirectional_lact_swiglu(*args, use_muon=False).double()
    want = _exact(*args)
    # fp32 throughout: a few roundings of sums of up to d and 64 terms, 2^-24 each
    assert (o - want).norm() <= 2e-6 * want.norm()


@pytest.mark.parametrize("power", [-59, -56, -53, -40, 20])
def test_small_queries(lb, power):
    """Gate and hidden activations near the smallest normal number keep their bits (hidden = about q^2)."""
    b, n, d, h = 2, 200, 64, 136
    w0, w1, w2, q, k, v, *lr = _inputs(b, n, d, h, seed=7)
    q = q * 2.0 ** power
    o = lb.block_causal_lact_swiglu(w0, w1, w2, q, k, v, *lr, chunk_size=256, use_muon=False).double()
    want = (F.silu(q.double() @ w0.double().mT) * (q.double() @ w2.double().mT)) @ w1.double().mT
    assert (o - want).norm() <= 2e-6 * want.norm()


# (what, times a power of two): the gradients of the weights, read as the momentum that starts at zero
@pytest.mark.parametrize("what,power", [("v", -116), ("v", -109), ("v", 118), ("lr", -116), ("lr", -109), ("k", -55), ("k", -50)])
def test_small_and_large_gradients(lb, what, power):
    b, n, d, h = 2, 200, 72, 128
    a = _inputs(b, n, d, h, seed=8)
    for i in {"k": (4,), "v": (5,), "lr": (6, 7, 8)}[what]:
        a[i] = a[i] * 2.0 ** power
    zeros = [torch.zeros_like(w) for w in a[:3]]
    r = lb.ar_fast_weight_swish_glu_weight_norm_mini_batch_inference_with_momentum(
        *a, 1.0, mini_batch_size=n, do_update=True, use_moun=False, fw_momentum=torch.ones(b, n, 1, device="cuda"),
        dw0_momentum=zeros[0], dw1_momentum=zeros[1], dw2_momentum=zeros[2], use_momentum=True)
    for got, want in zip(r[4:7], _gradients(*(t.double() for t in a))):
        assert (got.double() - want).norm() <= 2e-6 * want.norm()


def test_gate_far_below_zero(lb):
    """The sigmoid is a plain division: 1 / (1 + e^88) is a subnormal number, not zero."""
    b, n, d, h = 1, 40, 64, 64
    w0, w1, w2, q, k, v, *lr = _inputs(b, n, d, h, seed=6)
    w1 = w1.abs()
    w0[:, :, 0], w2[:, :, 0] = 1.0, 1e22
    q = torch.zeros_like(q)
    q[0, :, 0] = -torch.linspace(80, 88.5, n, device="cuda")   # what the gate sees
    o = lb.block_causal_lact_swiglu(w0, w1, w2, q, k, v, *lr, chunk_size=64, use_muon=False).double()
    want = (F.silu(q.double() @ w0.double().mT) * (q.double() @ w2.double().mT)) @ w1.double().mT
    # a subnormal sigmoid is a multiple of 2^-149 (and at least 2^-128); else an ulp or two of e^88
    assert ((o - want).abs() <= (2e-6 + 2.0 ** -22) * want.abs()).all()


def test_infinities_and_large_values(lb):
    """A token's infinity reaches its own outputs as an infinity, a NaN as a NaN, and no other token; values that bf16 rounds to
    infinity stay finite."""
    b, n, d, h = 2, 130, 64, 64
    w0, w1, w2, q, k, v, *lr = _inputs(b, n, d, h, seed=5)
    w0, w1, w2 = w0.abs(), w1.abs(), w2.abs()   # no sums of opposite infinities
    q = q.abs()
    apply = lambda x: lb.block_causal_lact_swiglu(w0, w1, w2, x, k, v, *lr, chunk_size=256, use_muon=False)
    plain = apply(q)
    x = q.clone()
    x[0, 3, 7] = float("inf")
    x[1, 64, 0] = float("nan")
    x[1, 129] = 3.4e38 * F.one_hot(torch.tensor(5), d).cuda()
    w0[:, :, 5] = w2[:, :, 5] = 1e-30
    plain, o = apply(q), apply(x)
    assert torch.isposinf(o[0, 3]).all() and torch.isnan(o[1, 64]).all()
    y = 3.4e38 * 1e-30
    want = (w1.double().sum(2) * (y * y))[1]
    assert ((o[1, 129].double() - want).abs() <= 1e-5 * want).all()
    same = torch.ones(b, n, dtype=torch.bool, device="cuda")
    same[0, 3] = same[1, 64] = same[1, 129] = False
    assert torch.equal(o[same], plain[same])
