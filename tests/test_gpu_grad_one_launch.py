"""The fast-weight gradient of heads of 128 features in one launch against the two launches, bit for bit: the way is chosen by the number
of entries, and an entry has the same bits in any batch; tokens whose learning rates are zero add nothing."""
import pytest
import torch

from launched_kernels import kernels

pytestmark = pytest.mark.gpu


def _inputs(b, n, h, lr_dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    d = 128
    w = [rn(b, h, d) / d ** 0.5, rn(b, d, h) / h ** 0.5, rn(b, h, d) / d ** 0.5]
    qkv = [torch.nn.functional.normalize(rn(b, n, d), dim=-1).bfloat16() for _ in range(2)] + [rn(b, n, d).bfloat16()]
    lrs = [torch.nn.functional.softplus(rn(b, n, 1) - 2.0).to(lr_dtype) for _ in range(3)]
    return w, qkv, lrs, torch.sigmoid(rn(b, n, 1)), [rn(*x.shape) for x in w]


def _step(w, qkv, lrs, gate, m, muon):
    import lact_b200 as lb
    n = qkv[0].shape[1]
    out = lb.ar_fast_weight_swish_glu_weight_norm_mini_batch_inference_with_momentum(
        *w, *qkv, *lrs, 1.0, mini_batch_size=n, do_update=True, use_moun=muon, num_moun_iters=5, fw_momentum=gate,
        dw0_momentum=m[0], dw1_momentum=m[1], dw2_momentum=m[2], use_momentum=True)
    lb.synchronize_and_check()
    return [t for t in out if torch.is_tensor(t)]


def _same(a, b):
    assert len(a) == len(b) >= 7
    for x, y in zip(a, b):
        assert torch.equal(x, y)


# an entry alone takes two launches at these lengths, sixteen take one: ends of tiles of 128 tokens, of k-blocks of 64, of both
@pytest.mark.parametrize("n", [2048, 2049, 2111, 2175, 2177, 2300, 4000])
@pytest.mark.parametrize("h,muon,lr", [(256, True, torch.float32), (128, False, torch.bfloat16)])
def test_entries_of_a_batch_and_alone(n, h, muon, lr):
    w, qkv, lrs, gate, m = _inputs(16, n, h, lr)
    both = _step(w, qkv, lrs, gate, m, muon)
    for e in (0, 7, 15):
        one = lambda ts: [t[e:e + 1].contiguous() for t in ts]
        _same([t[e:e + 1] for t in both], _step(one(w), one(qkv), one(lrs), gate[e:e + 1].contiguous(), one(m), muon))


# few tokens (one launch) against the same tokens in front of others whose learning rates are zero (two launches)
@pytest.mark.parametrize("n", [1, 5, 63, 64, 65, 127, 128, 129, 200, 256, 257, 385])
@pytest.mark.parametrize("h", [128, 256, 384])
def test_few_tokens_and_zero_learning_rates(n, h):
    w, qkv, lrs, gate, m = _inputs(1, 2300, h, torch.float32, seed=n)
    for t in lrs:
        t[:, n:] = 0
    gate[:] = gate[:, :1]      # (the momentum's factor is the mean gate of the tokens)
    gate = torch.full_like(gate, 0.5)
    few = _step(w, [t[:, :n].contiguous() for t in qkv], [t[:, :n].contiguous() for t in lrs], gate[:, :n].contiguous(), m, True)
    many = _step(w, qkv, lrs, gate, m, True)
    _same([t[:, :n] if t.dim() == 3 and t.shape[1] == 2300 else t for t in many], few)


def test_tokens_before_the_range_and_strided_rows():
    """An update of a later frame (the tile's rows begin inside the arrays) on rows that are views of a fused projection."""
    import lact_b200 as lb
    b, f, h = 12, 1560, 256
    w, _, lrs, gate, _ = _inputs(b, 3 * f, h, torch.float32, seed=3)
    g = torch.Generator(device="cuda").manual_seed(4)
    wide = torch.randn(b, 3 * f, 3 * 128, device="cuda", generator=g).bfloat16()
    q, k, v = (wide[..., i * 128:(i + 1) * 128] for i in range(3))
    run = lambda q, k, v, sel: lb.ar_fast_weight_swish_glu_weight_norm_mini_batch_with_momentum(
        *[t[sel] for t in w], q[sel], k[sel], v[sel], *[t[sel] for t in lrs], 1.0, mini_batch_size=f, update_every=f, use_moun=False,
        num_moun_iters=5, fw_momentum=gate[sel], use_momentum=True)
    views = run(q, k, v, slice(None))
    copies = run(q.contiguous(), k.contiguous(), v.contiguous(), slice(None))
    alone = run(q.contiguous(), k.contiguous(), v.contiguous(), slice(3, 4))
    lb.synchronize_and_check()
    for x, y, z in zip(views, copies, alone):
        assert torch.equal(x, y) and torch.equal(x[3:4], z)


# rows past the end of the last tile: their k and v are zeros, and zero times infinity is not
@pytest.mark.parametrize("n", [2049, 2111, 2177, 2304])
@pytest.mark.parametrize("h", [128, 256])
def test_infinite_weights(n, h):
    import lact_b200 as lb
    w, (_, k, v), lrs, _, _ = _inputs(16, n, h, torch.float32, seed=n)
    w02, w1, k, v = torch.cat([w[0], w[2]], 1).bfloat16(), w[1].bfloat16(), k.abs().clamp(min=2.0 ** -10), v.abs().clamp(min=2.0 ** -10)   # (no exact zeros)
    w02[:, 7] = w02[:, 7].abs()
    w1[:, 5, 7] = float("inf")      # dh of hidden feature 7 is +inf for every token, and so is dy2
    w02[:, h + 9, 3] = float("inf")   # y2 of hidden feature 9
    run = lambda s: lb.fused_lact_swiglu_ffn_fast_weight_grads(w02[s], w1[s], k[s], v[s], *[t[s, :, 0].contiguous() for t in lrs])
    both = run(slice(None))
    lb.synchronize_and_check()
    assert bool((both[0][:, h + 7] == float("inf")).all())
    for e in (0, 15):
        for x, y in zip(both, run(slice(e, e + 1))):
            assert torch.equal(x[e:e + 1].isnan(), y.isnan()) and torch.equal(x[e:e + 1].nan_to_num(), y.nan_to_num())


def _launches(call):
    """The kernels of the gradient that a call launches: "one" for both stages, "pointwise" and "contract" for one each."""
    return kernels(call, {"grad_gemm_kernel": "one", "OpFwGradPointwise": "pointwise", "OpDW": "contract"})


def _grads(w, qkv, lrs):
    import lact_b200 as lb
    w02, w1 = torch.cat([w[0], w[2]], 1).bfloat16(), w[1].bfloat16()
    lrs = [t[..., 0].contiguous() for t in lrs]
    return lb.fused_lact_swiglu_ffn_fast_weight_grads(w02, w1, qkv[1], qkv[2], *lrs)


# what is compared in this file: a batch that takes one launch, a few of its entries that take two.  More CTAs than SMs (clusters in a second
# round, full and nearly empty), as many clusters as fit, the most tokens that sixteen entries take in one launch
@pytest.mark.parametrize("b,n,h", [(32, 2048, 256), (48, 2177, 128), (24, 2300, 256), (16, 4000, 256), (64, 2049, 256), (37, 2111, 128),
                                   (16, 2048, 128), (16, 2300, 128)])
def test_one_launch_against_two(b, n, h):
    import lact_b200 as lb
    w, qkv, lrs, _, _ = _inputs(b, n, h, torch.float32, seed=b + n)
    both = _grads(w, qkv, lrs)
    assert _launches(lambda: _grads(w, qkv, lrs)) == ["one"]
    for e in (0, b // 2, b - 1):
        at = lambda ts: [t[e:e + 1].contiguous() for t in ts]
        alone = _grads(at(w), at(qkv), at(lrs))
        for x, y in zip(both, alone):
            assert torch.equal(x[e:e + 1], y)
    assert _launches(lambda: _grads(at(w), at(qkv), at(lrs))) == ["contract", "pointwise"]
    lb.synchronize_and_check()


# with momentum and Newton-Schulz, whose norms the launch leaves behind as partial sums: the second round of clusters too
@pytest.mark.parametrize("b,n,h", [(32, 2177, 256), (48, 2048, 128), (16, 4000, 256)])
def test_a_whole_update_with_more_ctas_than_sms(b, n, h):
    w, qkv, lrs, gate, m = _inputs(b, n, h, torch.float32, seed=n)
    both = _step(w, qkv, lrs, gate, m, True)
    assert _launches(lambda: _grads(w, qkv, lrs)) == ["one"]
    for e in (0, b // 2, b - 1):
        one = lambda ts: [t[e:e + 1].contiguous() for t in ts]
        _same([t[e:e + 1] for t in both], _step(one(w), one(qkv), one(lrs), gate[e:e + 1].contiguous(), one(m), True))


# few tokens: one launch on the side with few, two on the side with many
@pytest.mark.parametrize("n,ways", [(1, ["one"]), (128, ["one"]), (385, ["one"]), (2300, ["contract", "pointwise"])])
@pytest.mark.parametrize("h", [128, 256, 384])
def test_the_way_of_one_entry(n, ways, h):
    w, qkv, lrs, _, _ = _inputs(1, n, h, torch.float32)
    assert _launches(lambda: _grads(w, qkv, lrs)) == ways


# the faster way, both measured: chains in whole rounds of the SMs; a last round of few CTAs, few tokens per round, few CTAs
@pytest.mark.parametrize("b,n,h,one", [(12, 384, 256, True), (12, 1560, 256, True), (18, 5632, 128, True), (16, 4096, 128, True), (37, 780, 512, True),
                                       (37, 128, 256, True), (20, 16, 512, False), (40, 16, 256, False), (20, 16, 256, False), (40, 16, 128, False),
                                       (19, 780, 256, False), (38, 780, 128, False), (40, 384, 512, False), (28, 384, 512, False),
                                       (1, 2048, 256, False), (2, 1560, 256, False)])
def test_the_faster_way(b, n, h, one):
    w, qkv, lrs, _, _ = _inputs(b, n, h, torch.float32)
    assert _launches(lambda: _grads(w, qkv, lrs)) == (["one"] if one else ["contract", "pointwise"])
