"""Attention tiles cut over their keys (few query tiles, a short last round): outputs and log-sum-exps against whole tiles."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(L, q, k, v, window, cut, seq=None):
    b, l, h, d = q.shape
    lk = k.shape[1]
    o, lse = torch.full_like(q, float("nan")), torch.full((b, h, l), float("nan"), device="cuda")
    need, words = C.c_size_t(0), C.c_int64(0)
    if cut:
        L.check(L.lib().lact_swa_fwd_split_bytes(b, l, lk, h, d, window, C.byref(need), C.byref(words)), "split_bytes")
        assert need.value > 0
    scratch = torch.full((max(need.value, 256),), 0xFF, dtype=torch.uint8, device="cuda")   # NaNs: every word read was written
    counters = torch.zeros(max(words.value, 1), dtype=torch.int32, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    L.check(L.lib().lact_swa_fwd_split(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), b, l, lk, h, d, q.stride(1), q.stride(0),
                                       k.stride(1), k.stride(0), v.stride(1), v.stride(0), o.stride(1), o.stride(0), window, d ** -0.5,
                                       seq.data_ptr() if seq is not None else None, lse.data_ptr(),
                                       counters.data_ptr() if cut else None, scratch.data_ptr() if cut else None, need.value,
                                       status.data_ptr(), L.stream_ptr()), "swa")
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    return o, lse


# (entries, queries, keys, heads, d, window; window < 0: block attention): one query tile, fewer tiles than SMs, whole rounds
# and a short one, key counts that end inside a tile or leave a share empty, causal and banded tiles with fewer keys than shares
@pytest.mark.parametrize("b,l,lk,h,d,window", [(1, 1, 12481, 4, 64, -1), (1, 100, 4581, 4, 128, -1), (1, 1560, 4680, 12, 128, -1),
                                               (2, 129, 2291, 5, 64, -1), (1, 4680, 4681, 5, 128, -1), (1, 2500, 2500, 3, 128, 0),
                                               (2, 1155, 1155, 3, 64, 1100), (1, 2305, 2305, 8, 128, 2048)])
def test_split_equals_whole(b, l, lk, h, d, window):
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(l + lk)
    rn = lambda n: torch.randn(b, n, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = rn(l), rn(lk), rn(lk)
    if window < 0:
        k[:, : lk // 2] *= 3     # the running maximum lies in one share
    o, lse = _run(L, q, k, v, window, True)
    again, _ = _run(L, q, k, v, window, True)
    assert torch.equal(o, again)
    whole, lse_whole = _run(L, q, k, v, window, False)
    qf, kf, vf = (t.double().transpose(1, 2) for t in (q, k, v))
    s = qf @ kf.transpose(2, 3) * d ** -0.5
    if window >= 0:
        i, j = torch.arange(l, device="cuda")[:, None], torch.arange(lk, device="cuda")[None]
        s = s.masked_fill((j > i) | ((j <= i - window) if window > 0 else torch.zeros_like(j > i)), float("-inf"))
    want = (s.softmax(-1) @ vf).transpose(1, 2)
    err = lambda x: float((x.double() - want).norm() / want.norm())
    # probabilities and results are rounded to bf16 (2^-9 each) either way; the shares are combined in fp32
    assert err(o) <= 6e-3 and err(o) <= 1.02 * err(whole) + 1e-5
    assert float((lse - lse_whole).abs().max()) <= 1e-4    # log2 of a sum of exp2 approximations (2^-22 each)


def test_split_packed_sequences():
    from lact_b200 import _lib as L
    n, h, d = 1700, 4, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(1, n, h, d, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    seq = torch.zeros(n, dtype=torch.int32, device="cuda")
    seq[700:1500] = 700
    seq[1500:] = 1500
    o, _ = _run(L, q, k, v, 1024, True, seq)
    for s, e in ((0, 700), (700, 1500), (1500, n)):
        part, _ = _run(L, *(t[:, s:e].contiguous() for t in (q, k, v)), 1024, False)
        assert float((o[:, s:e].double() - part.double()).norm() / part.double().norm()) <= 4e-3   # bf16 probabilities and results
