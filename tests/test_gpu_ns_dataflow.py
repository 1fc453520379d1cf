"""Newton-Schulz by the dataflow kernel: sides that 256 divides, and results stored from registers by 64-, 128- and 192-wide and
symmetric tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lact_b200 import build
    build.build()
    import lact_b200
    from oracle import lact_oracle
    return lact_b200, lact_oracle


# (matrices: few select 64-wide tiles, 28 of side 256 or 7 of 512 the 128-wide ones, 19 of 512 the symmetric ones)
@pytest.mark.parametrize("nmat,R,C", [(28, 256, 256), (3, 768, 256), (7, 512, 512), (19, 512, 768), (2, 1024, 512),
                                      (38, 384, 384), (1, 136, 200), (3, 320, 328)])
@pytest.mark.parametrize("steps", [None, 1])
def test_sides_and_tiles(mods, nmat, R, C, steps):
    lb, orc = mods
    G = torch.randn(nmat, R, C, generator=torch.Generator().manual_seed(R + C))
    x = lb.zeropower_via_newtonschulz5(G.cuda(), steps).cpu()
    # at least as accurate as the reference's bf16 iteration (the slack of the parity test of this entry point)
    few = G[:2]
    ref, f64 = orc.newton_schulz(few, steps), orc.newton_schulz_f64(few, steps)
    assert orc.rel_fro(x[:2], f64) <= 1.25 * orc.rel_fro(ref, f64) + 2e-3
    # a matrix has the same bits in any batch, whatever tiles the batch selects
    assert torch.equal(lb.zeropower_via_newtonschulz5(G[-1:].cuda(), steps).cpu(), x[-1:])
