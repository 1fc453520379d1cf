"""The second-order pointwise stage at every head size with its own lane split, and next to them, with token counts that end
inside a block, against the formulas in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 56, 64, 72, 128, 192, 256, 320, 384, 512, 640])
@pytest.mark.parametrize("B,n,add", [(1, 1, False), (3, 37, True), (2, 64, False)])
def test_fw_grad_bwd_pointwise(H, B, n, add):
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(H + n)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    y, dh, gdy, ghid = rn(B, n, 2 * H), rn(B, n, H), rn(B, n, 2 * H), rn(B, n, H)
    lr = [torch.rand(B, n + 3, device="cuda", generator=g) for _ in range(3)]
    glr = [torch.ones(B, n + 5, device="cuda") for _ in range(3)]
    nan = lambda *s: torch.full(s, float("nan"), device="cuda", dtype=torch.bfloat16)
    gy, gdh, dy, hid = nan(B, n, 2 * H), nan(B, n, H), nan(B, n, 2 * H), nan(B, n, H)
    p = lambda t: t.data_ptr()
    L.check(L.lib().lact_fw_grad_bwd_pointwise(p(y), p(dh), p(gdy), p(ghid), p(lr[0]), p(lr[1]), p(lr[2]), L.dtype_code(lr[0]), 1.0,
                                               p(gy), p(gdh), p(dy), p(hid), p(glr[0]), p(glr[1]), p(glr[2]), B, n, H, n + 3, n + 5,
                                               int(add), L.stream_ptr()), "pointwise")
    torch.cuda.synchronize()
    y0, y2 = y.double().chunk(2, -1)
    d0, d2 = gdy.double().chunk(2, -1)
    h, gh = dh.double(), ghid.double()
    l0, l1, l2 = (t[:, :n, None].double() for t in lr)
    s = torch.sigmoid(y0)
    sw, A, Ap = s * y0, s * (1 + y0 * (1 - s)), s * (1 - s) * (2 + y0 * (1 - 2 * s))
    want = [torch.cat([gh * A * y2 * l1 + d0 * Ap * y2 * h * l0 + d2 * A * h * l2, gh * sw * l1 + d0 * A * h * l0], -1),
            d0 * A * y2 * l0 + d2 * sw * l2, torch.cat([A * y2 * h * l0, sw * h * l2], -1), sw * y2 * l1]
    # one rounding to bf16 (8 significant bits: at most 2^-8 of a value) of fp32 arithmetic with approximate sigmoids (1e-5)
    for got, w in zip((gy, gdh, dy, hid), want):
        assert float((got.double() - w).norm() / w.norm()) <= 2 ** -8 + 1e-5
    sums = [(d0 * A * y2 * h), (gh * sw * y2), (d2 * sw * h)]
    for got, w in zip(glr, sums):   # fp32 sums of H terms with approximate sigmoids (1e-6 each)
        err = (got[:, :n].double() - w.sum(-1) - (1 if add else 0)).abs()
        assert bool((err <= 1e-5 * (1 + w.abs().sum(-1))).all()) and bool((got[:, n:] == 1).all())
