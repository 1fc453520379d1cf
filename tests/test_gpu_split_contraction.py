"""Split token contractions: sums cut over several units per output tile, added in a fixed order by the last to arrive."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(L, a, b, c, accumulate):
    d = L.BmmDesc()
    d.a0, d.b0, d.c = a.data_ptr(), b.data_ptr(), c.data_ptr()
    d.a0_ld, d.a0_bs, d.b0_ld, d.b0_bs, d.c_ld, d.c_bs = a.stride(1), a.stride(0), b.stride(1), b.stride(0), c.stride(1), c.stride(0)
    d.batch, d.M, d.N, d.K = a.shape[0], a.shape[2], b.shape[2], a.shape[1]
    d.a0_mn = d.b0_mn = 1
    d.c_dtype, d.accumulate = L.dtype_code(c), int(accumulate)
    return d


# (entries, d, h, tokens, split): the shortest sum that is split, remainders of a k-block and of a unit, outputs narrower than
# a tile (72, 88), tiles of every width, more tiles than SMs, the longest sum; and the longest that stays whole
@pytest.mark.parametrize("entries,d,h,tokens,split", [(1, 64, 64, 6081, True), (2, 64, 64, 6080, False), (1, 128, 128, 6144, True),
                                                      (2, 192, 192, 6555, True), (1, 72, 88, 9999, True), (2, 384, 384, 8200, True),
                                                      (12, 128, 256, 6200, True), (1, 256, 256, 12289, True),
                                                      (3, 192, 192, 49152, True), (64, 64, 128, 6100, True)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_split_products(entries, d, h, tokens, split, accumulate):
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(entries * 1000 + tokens)
    x = [torch.randn(entries, tokens, n, device="cuda", generator=g).to(torch.bfloat16) for n in (2 * h, d, d, h)]
    c0 = [torch.randn(entries, 2 * h, d, device="cuda", generator=g), torch.randn(entries, d, h, device="cuda", generator=g)]
    counters = torch.zeros(512, dtype=torch.int32, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    results = []
    for _ in range(2):
        c = [t.clone() for t in c0]
        descs = (L.BmmDesc * 2)(_problem(L, x[0], x[1], c[0], accumulate), _problem(L, x[2], x[3], c[1], accumulate))
        need, words = C.c_size_t(0), C.c_int64(0)
        L.check(L.lib().lact_bmm_group_split_bytes(descs, 2, C.byref(need), C.byref(words)), "split_bytes")
        assert (need.value > 0) == split and words.value <= counters.numel()
        scratch = torch.full((max(need.value, 256),), 0xFF, dtype=torch.uint8, device="cuda")  # NaNs: every word read was written
        L.check(L.lib().lact_bmm_group_split_bf16(descs, 2, counters.data_ptr(), scratch.data_ptr(), need.value, status.data_ptr(),
                                                  L.stream_ptr()), "split")
        torch.cuda.synchronize()
        assert int(status[0]) == 0 and int(counters.abs().max()) == 0
        results.append(c)
    for i in range(2):
        assert torch.equal(results[0][i], results[1][i])
        want = x[2 * i].double().transpose(1, 2) @ x[2 * i + 1].double() + (c0[i].double() if accumulate else 0)
        # products of bf16 values are exact in fp32; n sums of them in fp32 lose at most n * 2^-24 of the terms' magnitudes,
        # about sqrt(n) * 2^-24 as the signs come: 1.3e-5 at 49152
        assert float((results[0][i].double() - want).norm() / want.norm()) <= 2e-5


# an entry's update is the same bits alone and in a batch
@pytest.mark.parametrize("d,h,tokens", [(192, 192, 6200), (128, 256, 8192)])
def test_split_update_is_independent_of_the_batch(d, h, tokens):
    import lact_b200 as lb
    g = torch.Generator(device="cuda").manual_seed(7)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    b = 40
    w = [rn(b, h, d) / d ** 0.5, rn(b, d, h) / h ** 0.5, rn(b, h, d) / d ** 0.5]
    qkv = [(lambda t: t / t.norm(dim=-1, keepdim=True))(rn(b, tokens, d)).to(torch.bfloat16) for _ in range(3)]
    args = w + qkv + [torch.rand(b, tokens, 1, device="cuda", generator=g) * 0.1 for _ in range(3)]
    whole = lb.bidirectional_lact_swiglu(*args, use_muon=True)
    assert torch.isfinite(whole).all()
    assert torch.equal(whole[17:18], lb.bidirectional_lact_swiglu(*[t[17:18].contiguous() for t in args], use_muon=True))
