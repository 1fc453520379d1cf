"""Attention tiles cut over their keys against whole tiles on values that are not finite: NaN and infinite rows and keys reach
the same outputs and log-sum-exps, and the rows they do not reach are untouched."""
import pytest
import torch

from test_gpu_swa_split import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,l,lk,h,d,window", [(1, 100, 4581, 4, 128, -1), (1, 1560, 4680, 12, 128, -1), (2, 129, 2291, 5, 64, -1),
                                               (1, 2305, 2305, 8, 128, 2048)])
@pytest.mark.parametrize("where", ["query", "key", "value", "all"])
def test_cut_tiles_keep_nan_and_inf(b, l, lk, h, d, window, where):
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(l + lk)
    rn = lambda n: torch.randn(b, n, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = rn(l), rn(lk), rn(lk)
    nan, inf = float("nan"), float("inf")
    if where == "query":      # one element of a row: every score of the row; rows of the first and of the last tile
        q[:, 5, 0, 3] = nan
        q[:, 7, 1, 0] = inf
        q[:, -1, 2] = nan
        q[:, -2, 3] = -inf
    elif where == "key":      # scores of one share
        k[:, lk - 300, 0] = nan
        k[:, lk - 290, 1, 0] = inf
        k[:, 40, 2, 1] = -inf
    elif where == "value":
        v[:, lk - 300, 0] = nan
        v[:, lk - 290, 1, 0] = inf
    else:                     # a run that has diverged as a whole
        q[:], k[:] = nan, nan
    o, lse = _run(L, q, k, v, window, True)
    ow, lsew = _run(L, q, k, v, window, False)
    for cut, whole in ((o.float(), ow.float()), (lse, lsew)):
        assert torch.equal(cut.isnan(), whole.isnan())
        assert torch.equal(cut.nan_to_num(0.0, 0.0, 0.0) == 0, whole.nan_to_num(0.0, 0.0, 0.0) == 0)
        assert torch.equal(cut[cut.isinf()], whole[cut.isinf()])
    ok = o.isfinite()
    if ok.any():   # bf16 results of sums in another order: one rounding (2^-9) each
        assert float((o[ok].double() - ow[ok].double()).norm()) <= 4e-3 * float(ow[ok].double().norm())


# (tokens, window, query, key): a query past the band of the keys 0 to 127 in the last tile they meet, a key before the band of a
# query tile in the first tile it meets
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("l,window,row,key", [(1024, 64, 224, 150), (1024, 64, 192, 191), (700, 33, 170, 351), (900, 200, 352, 303),
                                              (640, 130, 288, 100)])
def test_gradients_past_the_band_stay_finite(d, l, window, row, key):
    """128 rows of one side meet a group of 16 rows of the other or they do not: a gradient or a value that is not finite reaches
    the tiles whose band its group is in, and in all others the gradients keep their bits."""
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(l + row)
    rn = lambda: torch.randn(1, l, 2, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v, do = rn(), rn(), rn(), rn()
    fwd, lse = _run(L, q, k, v, window, False)

    def grads(v, do):
        out = [torch.empty_like(q) for _ in range(3)]
        delta, status = torch.empty_like(lse), torch.zeros(64, dtype=torch.int32, device="cuda")
        L.check(L.lib().lact_swa_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), fwd.data_ptr(), do.data_ptr(), lse.data_ptr(),
                                     *[t.data_ptr() for t in out], delta.data_ptr(), 1, l, l, 2, d, *[2 * d, 2 * d * l] * 5, window,
                                     d ** -0.5, None, status.data_ptr(), L.stream_ptr()), "bwd")
        torch.cuda.synchronize()
        assert int(status[0]) == 0
        return out

    def with_row(t, i, value):
        t = t.clone()
        t[:, i] = value
        return t

    clean = grads(v, do)
    group = lambda i: (i // 16 * 16, i // 16 * 16 + 15)
    tiles = range(0, l, 128)
    _, dk, dv = grads(v, with_row(do, row, float("nan")))
    free = [o for o in tiles if group(row)[0] > o + 127 + window - 1 or group(row)[1] < o]
    assert 0 in free
    for o in free:
        assert torch.equal(dk[:, o:o + 128], clean[1][:, o:o + 128]) and torch.equal(dv[:, o:o + 128], clean[2][:, o:o + 128])
    dq, _, _ = grads(with_row(v, key, float("inf")), do)
    free = [o for o in tiles if group(key)[1] < o - (window - 1) or group(key)[0] > o + 127]
    assert any(key // 128 == (o - (window - 1)) // 128 for o in free)
    for o in free:
        assert torch.equal(dq[:, o:o + 128], clean[0][:, o:o + 128])
