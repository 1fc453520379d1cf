"""Gradients of step programs whose token ranges overlap in part or lie inside one another, with the allocator's free memory
full of NaNs, against autograd through the CPU oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
NAMES = ("w0", "w1", "w2", "q", "k", "v", "lr0", "lr1", "lr2")


def fill_free_memory():
    """Leaves NaN bit patterns in the free blocks the next allocations are served from."""
    torch.cuda.empty_cache()
    junk = [torch.full((n,), 255, dtype=torch.uint8, device="cuda") for n in (1 << 21, 1 << 19, 1 << 16, 1 << 13, 512) for _ in range(48)]
    torch.cuda.synchronize()
    del junk


@pytest.mark.parametrize("order", [
    [(0, 100, True, False), (50, 150, True, False), (0, 120, False, True), (90, 192, False, True)],      # in part
    [(0, 150, True, False), (0, 64, True, False), (0, 192, False, True), (100, 150, False, True)],       # a prefix, a middle
    [(60, 90, True, False), (0, 192, True, True), (30, 70, True, True), (64, 192, False, True)],         # both sides stick out
])
def test_overlapping_update_and_apply_ranges(order):
    import lact_b200 as lb
    from oracle import lact_oracle as orc
    B, L, D, H = 2, 192, 64, 64
    i = orc.make_inputs(B, L, D, H, seed=11, act_dtype=BF16)
    for n in ("w0", "w1", "w2"):   # this driver keeps its weights transposed
        i[n] = i[n].transpose(1, 2).contiguous()
    n_out = sum(e - s for s, e, _, a in order if a)
    dO = torch.randn(B, n_out, D, generator=torch.Generator().manual_seed(4)).to(BF16)
    ref = {n: i[n].float().clone().requires_grad_(True) for n in NAMES}
    orc.nvs_mini_batch_apply(*[ref[n] for n in NAMES], order, 0)[0].backward(dO.float())
    got = {n: i[n].cuda().requires_grad_(True) for n in NAMES}
    o = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*[got[n] for n in NAMES], order)[0]
    d = dO.cuda()
    fill_free_memory()
    o.backward(d)
    lb.synchronize_and_check()
    for n in NAMES:
        a, b = got[n].grad.float().cpu(), ref[n].grad.float()
        assert torch.isfinite(a).all(), n
        # bf16 operands in the backward's products (2^-9 each, a few of them in a row)
        assert orc.rel_max(a, b) <= 3e-2 and orc.cosine(a, b) >= 0.999, (n, orc.rel_max(a, b))


def test_outputs_that_a_later_apply_overwrites():
    """num_repeat > 1 applies every token range once per repetition and keeps the last result: earlier ones have no gradient."""
    import lact_b200 as lb
    from oracle import lact_oracle as orc
    B, L, D, H = 2, 256, 64, 64
    i = orc.make_inputs(B, L, D, H, seed=13, act_dtype=BF16)
    dO = torch.randn(B, L, D, generator=torch.Generator().manual_seed(6)).to(BF16)
    kw = dict(num_repeat=2, mini_batch_size=64, update_every=64)
    ref = {n: i[n].float().clone().requires_grad_(True) for n in NAMES}
    orc.ar_mini_batch(*[ref[n] for n in NAMES], 1.0, **kw)[0].backward(dO.float())
    got = {n: i[n].cuda().requires_grad_(True) for n in NAMES}
    o = lb.ar_fast_weight_swish_glu_weight_norm_mini_batch(*[got[n] for n in NAMES], 1.0, **kw)[0]
    d = dO.cuda()
    fill_free_memory()
    o.backward(d)
    lb.synchronize_and_check()
    for n in NAMES:
        a, b = got[n].grad.float().cpu(), ref[n].grad.float()
        assert orc.rel_max(a, b) <= 3e-2 and orc.cosine(a, b) >= 0.999, (n, orc.rel_max(a, b))


def test_outputs_overwritten_in_part():
    """Against the same program whose applies stop where a later one writes."""
    import lact_b200 as lb
    from lact_b200 import ops
    from lact_b200 import program as P
    from oracle import lact_oracle as orc
    i = orc.make_inputs(2, 192, 64, 64, seed=17, act_dtype=BF16)
    leaves = [i[n].cuda().requires_grad_(True) for n in NAMES]
    A, U = P.APPLY, P.UPDATE
    d = torch.randn(2, 192, 64, generator=torch.Generator().manual_seed(8)).to(BF16).cuda()
    grads = []
    for steps in ([(A, 0, 192, 0), (U, 0, 64, 0), (A, 40, 100, 60), (U, 64, 150, 0), (A, 100, 150, 100)],
                  [(A, 0, 60, 0), (A, 150, 192, 150), (U, 0, 64, 0), (A, 40, 80, 60), (U, 64, 150, 0), (A, 100, 150, 100)]):
        o = ops.scan(*leaves, steps)
        fill_free_memory()
        grads.append((o.detach(), *torch.autograd.grad(o, leaves, d)))
    lb.synchronize_and_check()
    for a, b in zip(*grads):   # the same values; bf16 products of other shapes, their sums in another order
        assert orc.rel_max(a.float().cpu(), b.float().cpu()) <= 2e-2
