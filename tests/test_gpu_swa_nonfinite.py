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
