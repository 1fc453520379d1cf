"""APPLY steps that wait for the last of their run and share one launch: the same bits as steps that run one by one.

A run ends where two APPLY steps follow each other without an update in between, or where the next one has another length, so the
same operators with a short APPLY of another length behind each of them run singly."""
import pytest
import torch

import lact_b200 as lb

pytestmark = pytest.mark.gpu


def _inputs(b, n, d, h, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    w = [rn(b, d, h) / d ** 0.5, rn(b, h, d) / h ** 0.5, rn(b, d, h) / d ** 0.5]
    q, k, v = (rn(b, n, d).to(torch.bfloat16) for _ in range(3))
    return w + [q, k, v] + [0.1 * rn(b, n, 1).abs() for _ in range(3)]


# tails of 128- and 256-row tiles; runs shorter than, as long as and longer than what one launch takes (64 entries of 300
# tokens and 256 features: 384 tiles a step, five steps a launch); pairs of SMs (24 entries of 384, two steps: 3 per launch)
@pytest.mark.parametrize("b,d,h,length,steps,muon", [
    (2, 64, 64, 1, 2, 5), (2, 64, 64, 1, 3, 0), (3, 128, 256, 129, 3, 0), (1, 192, 192, 300, 4, 5), (64, 128, 256, 300, 7, 0), (24, 384, 384, 640, 3, 0),
    (2, 80, 48, 257, 5, 0),
])
@pytest.mark.parametrize("train", [False, True])
def test_runs_equal_single_steps(b, d, h, length, steps, muon, train):
    if train and muon and d == 64:
        muon = 0
    args = _inputs(b, length * steps, d, h)
    if train:
        args = [a.requires_grad_(True) for a in args]
    op = lb.TTTOperator
    run, single = [], []
    extra = 1 if length != 1 else 2
    for i in range(steps):
        here = op(i * length, (i + 1) * length, True, True)
        run.append(here)
        single += [here, op(0, extra, False, True)]
    got = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*args, run, muon_update_steps=muon)
    want = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*args, single, muon_update_steps=muon)
    keep = torch.cat([torch.arange(i * (length + extra), i * (length + extra) + length) for i in range(steps)]).cuda()
    assert torch.equal(got[0], want[0][:, keep])
    for x, y in zip(got[1:], want[1:]):
        assert torch.equal(x, y)


def test_uneven_steps_stay_in_order():
    """Steps of other lengths or spacings end a run; what they write stays where it was."""
    b, d, h = 2, 128, 128
    args = _inputs(b, 1000, d, h, seed=1)
    op = lb.TTTOperator
    spans = [(0, 200), (200, 400), (400, 600), (650, 850), (850, 1000)]
    run = [op(s, e, True, True) for s, e in spans]
    single = [x for s, e in spans for x in (op(s, e, True, True), op(s, s + 1, False, True))]
    got = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*args, run, muon_update_steps=0)[0]
    want = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*args, single, muon_update_steps=0)[0]
    at = 0
    for i, (s, e) in enumerate(spans):
        assert torch.equal(got[:, at:at + e - s], want[:, at + i:at + i + e - s])
        at += e - s


# Steps of one length, evenly spaced, in which APPLY steps also follow each other directly: a run may begin in any slot of the
# weights and ends with the last one there is.
@pytest.mark.parametrize("program", ["UA UA A UA", "A UA A UA", "UA A UA A UA", "A A UA UA", "UA UA A UA UA A UA UA UA A UA UA",
                                     "A UA UA UA U UA A A UA UA UA UA"])
@pytest.mark.parametrize("b,d,h,length,muon", [(2, 64, 64, 130, 5), (3, 128, 256, 1, 0), (24, 384, 384, 256, 0), (48, 512, 512, 128, 0)])
@pytest.mark.parametrize("train", [False, True])
def test_runs_from_any_slot(program, b, d, h, length, muon, train):
    if train:
        muon = 0
    ops = program.split()
    args = _inputs(b, length * len(ops), d, h, seed=2)
    if train:
        args = [a.requires_grad_(True) for a in args]
    op = lb.TTTOperator
    extra = 1 if length != 1 else 2
    run, single, keep, at = [], [], [], 0
    for i, what in enumerate(ops):
        here = op(i * length, (i + 1) * length, "U" in what, "A" in what)
        run.append(here)
        single.append(here)
        if "A" in what:
            single.append(op(0, extra, False, True))
            keep.append(torch.arange(at, at + length))
            at += length + extra
    got = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*args, run, muon_update_steps=muon)
    want = lb.fast_weight_swish_glu_weight_norm_mini_batch_apply(*args, single, muon_update_steps=muon)
    lb.synchronize_and_check()
    assert torch.equal(got[0], want[0][:, torch.cat(keep).cuda()])
    for x, y in zip(got[1:], want[1:]):
        assert torch.equal(x, y)
