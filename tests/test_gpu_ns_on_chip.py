"""Newton-Schulz by one CTA per matrix (matrices that fit an SM) at the edges of its tiles: smallest and largest sides, one
and two 128-row tiles, tall updates in one and two passes, more matrices than SMs; kept iterates; the fallback just past
the limits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.fixture(scope="module")
def mods():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lact_b200 import build
    build.build()
    import lact_b200
    from lact_b200 import backward
    from oracle import lact_oracle
    return lact_b200, backward, lact_oracle


@pytest.mark.parametrize("nmat,R,C", [
    (1, 64, 64), (2, 64, 512), (2, 512, 64), (3, 128, 128), (2, 128, 256), (2, 256, 128), (1, 128, 512), (1, 448, 128),
    (2, 192, 192), (1, 192, 256), (2, 384, 192), (1, 64, 192), (1, 192, 64), (150, 64, 128),
    (1, 192, 320),    # wide and past 512 accumulator columns: the dataflow kernel
    (1, 96, 192),     # not a multiple of 64: the dataflow kernel
])
@pytest.mark.parametrize("steps", [None, 1, 4])
def test_newton_schulz_edges(mods, nmat, R, C, steps):
    lb, bw, orc = mods
    G = torch.randn(nmat, R, C, generator=torch.Generator().manual_seed(R + C))
    G[0] *= 1e3  # the normalisation is per matrix
    x = lb.zeropower_via_newtonschulz5(G.cuda(), steps).cpu()
    ref, f64 = orc.newton_schulz(G, steps), orc.newton_schulz_f64(G, steps)
    # at least as accurate as the reference's bf16 iteration (same slack as the parity test of this entry point)
    assert orc.rel_fro(x, f64) <= 1.25 * orc.rel_fro(ref, f64) + 2e-3
    assert torch.equal(lb.zeropower_via_newtonschulz5(G.to(BF16).cuda(), steps).cpu(), x)
    # every iterate kept (what training does): the same result, and the kept matrices reproduce it
    saved, U = bw.ns_forward_saved(G.cuda(), 5 if steps is None else steps, steps is not None, False)
    assert torch.equal(U.cpu(), x)
    dU = torch.randn(nmat, R, C, generator=torch.Generator().manual_seed(1)).to(BF16)
    got = bw.ns_backward(saved, dU.cuda()).double().cpu()
    bw.check_status(torch.device("cuda", 0))
    Gd = G.to(BF16).double().requires_grad_(True)
    f = orc.newton_schulz_f64
    X = Gd / (Gd.flatten(1).norm(dim=1).view(-1, 1, 1) + 1e-7)
    for a, b, c in (orc.NS_TUNED5 if steps is None else (orc.NS_CONST,) * steps):
        A = X @ X.transpose(1, 2) if R <= C else X.transpose(1, 2) @ X
        P = a * torch.eye(A.shape[1], dtype=torch.double) + b * A + c * A @ A
        X = P @ X if R <= C else X @ P
    (X * dU.double()).sum().backward()
    # bf16 operands through up to 15 products: the bands of the Newton-Schulz backward tests
    assert orc.cosine(got, Gd.grad) >= (0.995 if steps is None or steps > 1 else 0.9995)
