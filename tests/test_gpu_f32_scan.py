"""fp32 mode's recurrence (`lact_scan_f32_fwd`) at sizes where its 128 x 64 (128 x 32 fused) tiles, its k-slabs of 16 and
its token splits end in remainders, against the fp32 oracle (Muon off)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NAMES = ("w0", "w1", "w2", "q", "k", "v", "lr0", "lr1", "lr2")


@pytest.mark.parametrize("B,L,D,H,chunk", [
    (1, 9, 4, 8, 4),          # smallest head, chunks shorter than a k-slab
    (2, 131, 12, 40, 64),     # everything ragged
    (1, 259, 132, 136, 129),  # one past the tile edge in tokens, rows and columns
    (3, 1025, 64, 32, 1024),  # one token after a long, split contraction
    (17, 300, 192, 96, 263),  # many entries: no splits
])
@pytest.mark.parametrize("momentum", [False, True])
def test_f32_scan_remainders(B, L, D, H, chunk, momentum):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lact_b200 import build
    build.build()
    import lact_b200 as lb
    from oracle import lact_oracle as orc
    i = orc.make_inputs(B, L, D, H, seed=L)
    m = i["momentum"] if momentum else None
    want = orc.block_causal_lact_swiglu(*[i[n] for n in NAMES], chunk_size=chunk, use_muon=False, momentum=m)
    # a strided q: a view into a wider projection (token stride 2 D)
    wide = torch.zeros(B, L, 2 * D, device="cuda")
    wide[..., D:] = i["q"].cuda()
    c = {n: i[n].cuda() for n in NAMES}
    c["q"] = wide[..., D:]
    got = lb.block_causal_lact_swiglu(*[c[n] for n in NAMES], chunk_size=chunk, use_muon=False,
                                      momentum=m.cuda() if momentum else None)
    lb.synchronize_and_check()
    assert got.dtype == torch.float32
    # fp32 sums of at most 1024 terms: 1024 * 2^-24 = 6e-5 per product in the worst case (their square root in practice)
    assert orc.rel_max(got.cpu(), want) <= 1e-4
