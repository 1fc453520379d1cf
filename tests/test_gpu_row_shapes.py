"""The layer's row passes at every head size that has a lane split of its own, and next to them, with token counts that end
inside a block: forward and backward against the plain formulas in fp32."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _heads(x, n):
    b, s, nd = x.shape
    return x.reshape(b, s, n, nd // n).transpose(1, 2).reshape(b * n, s, nd // n)


def _close(got, want, tol):
    """|error| against the row's own scale: bf16 results of fp32 arithmetic (2^-9 each for the rounded SiLU, the rounded
    norm and the result; `tol` adds them up)."""
    got, want = got.float(), want.float()
    assert float((got - want).abs().max() / want.abs().max()) <= tol
    assert float((got - want).norm() / want.norm()) <= tol


@pytest.mark.parametrize("d,hd", [(64, 64), (128, 32), (192, 64), (256, 256), (384, 128), (512, 512), (768, 256), (1024, 1024),
                                  (320, 64), (72, 0)])
@pytest.mark.parametrize("b,s,n_h", [(2, 33, 3), (1, 1, 1)])
def test_row_passes(d, hd, b, s, n_h):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lact_b200 import build
    build.build()
    from lact_b200 import layer_ops as lo
    g = torch.Generator(device="cuda").manual_seed(d + s)
    rn = lambda *sh: torch.randn(*sh, device="cuda", generator=g).to(BF16)
    x = [rn(b, s, n_h * d).requires_grad_() for _ in range(3)]
    dz = [rn(b * n_h, s, d) for _ in range(3)]
    tables = (*lo.rotary_tables(hd, s + 2, device="cuda"), hd) if hd else None
    out = lo.qkv_prologue(*x, n_h, rotary=tables, seqlen_offset=2 if hd else 0)
    grads = torch.autograd.grad(out, x, dz)
    for i in range(3):
        xr = x[i].detach().float().requires_grad_()
        y = F.silu(_heads(xr, n_h))
        if i < 2:
            y = y / (y.norm(dim=-1, keepdim=True) + 1e-5)
            if hd:
                y = y.reshape(b * n_h, s, d // hd, hd)
                c, sn = (t[2:, None].float() for t in tables[:2])
                y1, y2 = y[..., :hd // 2], y[..., hd // 2:]
                y = torch.cat([y1 * c - y2 * sn, y1 * sn + y2 * c], dim=-1).reshape(b * n_h, s, d)
        _close(out[i], y.detach(), 4 * 2.0 ** -8)
        _close(grads[i], torch.autograd.grad(y, xr, dz[i].float())[0], 6 * 2.0 ** -8)
    fw, gate, res, w = rn(b * n_h, s, d), rn(b, s, n_h * d), rn(b, s, n_h * d), 1 + 0.1 * rn(d).float()
    dy = rn(b, s, n_h * d)
    leaves = [t.detach().clone().requires_grad_() for t in (fw, w, gate, res)]
    o = lo.out_epilogue(leaves[0], leaves[1], n_h, leaves[2], leaves[3])
    got = torch.autograd.grad(o, leaves, dy)
    ref = [t.detach().float().requires_grad_() for t in (fw, w, gate, res)]
    n = ref[0] * torch.rsqrt(ref[0].pow(2).mean(-1, keepdim=True) + 1e-5) * ref[1]
    n = n.reshape(b, n_h, s, d).transpose(1, 2).reshape(b, s, n_h * d)
    want_o = n * F.silu(ref[2]) + ref[3]
    _close(o.detach(), want_o.detach(), 4 * 2.0 ** -8)
    for a, r in zip(got, torch.autograd.grad(want_o, ref, dy.float())):
        _close(a, r, 4 * 2.0 ** -8)
