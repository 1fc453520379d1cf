"""Block attention over a cache and new keys, each where it lies: lengths around the key tiles, views, cut tiles, gradients."""
import pytest
import torch

from lact_b200 import layer_ops as lo

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _rows(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g).to(BF16)


def _want(q, k, v):
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * q.shape[3] ** -0.5
    return torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), v.double())


# a run of keys shorter than, as long as and just past a tile of 128, on either side; few query tiles (cut over their keys, more
# shares than some run has tiles) and many
@pytest.mark.parametrize("b,l,cached,new,h,d", [(1, 1, 1, 1, 4, 64), (2, 130, 127, 130, 4, 128), (1, 100, 128, 256, 8, 64),
                                                (1, 300, 1500, 1, 4, 128), (2, 129, 129, 1000, 4, 64), (1, 2500, 257, 300, 16, 128)])
def test_like_one_array(b, l, cached, new, h, d):
    g = torch.Generator(device="cuda").manual_seed(l + cached)
    q, k, v = _rows(g, b, l, h, d), _rows(g, b, new, h, d), _rows(g, b, new, h, d)
    cache = _rows(g, 2 * b, cached, h, d)
    o = lo.sliding_window_attention_inference(q, k, v, new, kv_cache=cache).double()
    kc, vc = cache.chunk(2)
    want = _want(q, torch.cat([kc, k], 1), torch.cat([vc, v], 1))
    # probabilities and output rounded to bf16 once each (2^-9), sums in fp32
    assert (o - want).norm() <= 4e-3 * want.norm()
    one = lo.block_attention(q, torch.cat([kc, k], 1), torch.cat([vc, v], 1)).double()
    assert (one - want).norm() <= 4e-3 * want.norm() and (o - one).norm() <= 4e-3 * want.norm()


def test_views_large_scores_and_gradients():
    g = torch.Generator(device="cuda").manual_seed(3)
    b, l, h, d = 2, 200, 4, 64
    qkv = _rows(g, b, l, 3 * h * d).view(b, l, 3, h, d)
    q, k, v = (qkv[:, :, i] for i in range(3))
    cache = 8 * _rows(g, 2 * b, 70, h, d)
    o = lo.sliding_window_attention_inference(q, k, v, l, kv_cache=cache)
    kc, vc = cache.chunk(2)
    want = _want(q, torch.cat([kc, k], 1), torch.cat([vc, v], 1))
    assert (o.double() - want).norm() <= 4e-3 * want.norm()
    # with gradients: those of attention over one array
    leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v, cache)]
    dout = _rows(g, b, l, h, d)
    got = torch.autograd.grad(lo.sliding_window_attention_inference(*leaves[:3], l, kv_cache=leaves[3]), leaves, dout)
    kc, vc = leaves[3].chunk(2)
    ref = torch.autograd.grad(lo.block_attention(leaves[0], torch.cat([kc, leaves[1]], 1), torch.cat([vc, leaves[2]], 1)), leaves, dout)
    assert all(torch.equal(x, y) for x, y in zip(got, ref))


def test_a_nan_key_reaches_every_query_of_its_head():
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v = (_rows(g, 1, 150, 4, 64) for _ in range(3))
    cache = _rows(g, 2, 130, 4, 64)
    cache[0, 129, 1, 0] = float("nan")
    o = lo.sliding_window_attention_inference(q, k, v, 150, kv_cache=cache)
    bad = torch.isnan(o).all(-1)
    assert bad[:, :, 1].all() and not torch.isnan(o[:, :, [0, 2, 3]]).any()
