"""Attention forward on pairs of query tiles: outputs and log-sum-exps against 64-bit attention where the pairs, the dealing of items to
SMs and the cut of the last ones have their edges."""
import pytest
import torch

from launched_kernels import kernels
from test_gpu_swa_split import _run

pytestmark = pytest.mark.gpu


def _kernels(call):
    """The attention kernels that a call launches."""
    return set(kernels(call, {"swa_pairs_kernel": "pairs", "swa_combine_kernel": "combine", "swa_fwd_kernel": "single"}))


def _prepared(q, k, v, window, cut, starts=None, failed=False):
    """A call of the C interface with all that it takes in hand; outputs filled with 7, and its status word."""
    import ctypes as C
    from lact_b200 import _lib as L
    b, l, h, d = q.shape
    lk = k.shape[1]
    o, lse = torch.full_like(q, 7.0), torch.full((b, h, l), 7.0, device="cuda")
    need, words = C.c_size_t(0), C.c_int64(0)
    L.check(L.lib().lact_swa_fwd_split_bytes(b, l, lk, h, d, window, C.byref(need), C.byref(words)), "split_bytes")
    scratch = torch.full((max(need.value, 256),), 0xFF, dtype=torch.uint8, device="cuda")
    counters = torch.zeros(max(words.value, 1), dtype=torch.int32, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    status[0] = 101 if failed else 0
    call = lambda: L.check(L.lib().lact_swa_fwd_split(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), b, l, lk, h, d, h * d, h * d * l, *[h * d, h * d * lk] * 2, h * d, h * d * l,
        window, d ** -0.5, starts.data_ptr() if starts is not None else None, lse.data_ptr(), counters.data_ptr() if cut else None,
        scratch.data_ptr() if cut else None, need.value, status.data_ptr(), L.stream_ptr()), "swa")
    return call, o, lse, status


def _reference(q, k, v, window, starts=None):
    l, lk, d = q.shape[1], k.shape[1], q.shape[-1]
    qf, kf, vf = (t.double().transpose(1, 2) for t in (q, k, v))
    s = qf @ kf.transpose(2, 3) * d ** -0.5
    if window >= 0:
        i, j = torch.arange(l, device="cuda")[:, None], torch.arange(lk, device="cuda")[None]
        hidden = j > i
        if window > 0:
            hidden |= j <= i - window
        if starts is not None:
            hidden |= j < starts[:, None]
        s = s.masked_fill(hidden, float("-inf"))
    return (s.softmax(-1) @ vf).transpose(1, 2), torch.logsumexp(s, -1) * 1.4426950408889634


def _compare(q, k, v, window, cut, starts=None):
    from lact_b200 import _lib as L
    o, lse = _run(L, q, k, v, window, cut, starts)
    want, want_lse = _reference(q, k, v, window, starts)
    assert torch.isfinite(o.float()).all()
    # probabilities and results are rounded to bf16 (2^-9 each)
    assert float((o.double() - want).norm() / want.norm()) <= 6e-3
    # the scores' products are summed in fp32 (2^-24 each over d terms), the exponentials are good to 2^-22
    assert float((lse.double() - want_lse).abs().max()) <= 1e-4


# one tile and two, rows on both sides of a tile's and a pair's end, windows that end on tiles and inside them (300 heads: calls with
# few tiles run on single ones)
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("l,window", [(1, 0), (127, 40), (128, 128), (129, 1), (255, 0), (256, 128), (257, 129), (385, 256), (511, 130),
                                      (513, 600)])
def test_ends_of_pairs(l, window, d):
    g = torch.Generator(device="cuda").manual_seed(l * 7 + window)
    q, k, v = (torch.randn(1, l, 300, d, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    _compare(q, k, v, window, False)


# more items than SMs: whole rounds and a rest that is cut; one round exactly; keys of block attention on both sides of a tile's end
@pytest.mark.parametrize("b,l,lk,h,d,window,cut", [(1, 1100, 1100, 40, 128, 0, False), (1, 2600, 2500, 14, 128, -1, True),
                                                   (2, 1900, 2600, 10, 64, -1, True),
                                                   (1, 257, 257, 74, 64, 200, False), (1, 300, 1025, 80, 128, -1, False),
                                                   (3, 130, 127, 30, 64, -1, False)])
def test_items_over_the_chip(b, l, lk, h, d, window, cut):
    g = torch.Generator(device="cuda").manual_seed(l + h)
    rn = lambda n: torch.randn(b, n, h, d, device="cuda", generator=g).to(torch.bfloat16)
    _compare(rn(l), rn(lk), rn(lk), window, cut)


@pytest.mark.parametrize("l,h,window,cut", [(1100, 60, 300, False), (2305, 8, 2048, True)])
@pytest.mark.parametrize("cuts", [(128, 256, 400), (1, 2, 383), (255, 257, 1000), (64, 640, 896)])
def test_packed_sequences_across_pairs(l, h, window, cut, cuts):
    g = torch.Generator(device="cuda").manual_seed(sum(cuts))
    q, k, v = (torch.randn(1, l, h, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    starts = torch.zeros(l, dtype=torch.int32, device="cuda")
    for c in cuts:
        starts[c:] = c
    _compare(q, k, v, window, cut, starts)


def test_growing_scores_reach_every_row():
    """Scores that grow along the keys: the maximum changes in every tile, for some rows by more than fp32's range of exponents."""
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(1, 900, 100, 64, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    k = (k * torch.linspace(0.1, 30, 900, device="cuda")[None, :, None, None]).to(torch.bfloat16)
    from lact_b200 import _lib as L
    o, _ = _run(L, q, k, v, 0, False)
    want, _ = _reference(q, k, v, 0)
    # one probability of 1 beside small ones: the result is that value's bf16 rounding or near it
    assert float((o.double() - want).norm() / want.norm()) <= 6e-3


@pytest.mark.parametrize("l,h,window,cut", [(300, 200, 0, False), (2305, 8, 2048, True)])
def test_nothing_is_written_after_an_earlier_failure(l, h, window, cut):
    import ctypes as C
    from lact_b200 import _lib as L
    b, d = 1, 128
    q, k, v = (torch.randn(b, l, h, d, device="cuda").to(torch.bfloat16) for _ in range(3))
    o, lse = torch.full_like(q, 7.0), torch.full((b, h, l), 7.0, device="cuda")
    need, words = C.c_size_t(0), C.c_int64(0)
    L.check(L.lib().lact_swa_fwd_split_bytes(b, l, l, h, d, window, C.byref(need), C.byref(words)), "split_bytes")
    scratch = torch.zeros(max(need.value, 256), dtype=torch.uint8, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    status[0] = 101
    L.check(L.lib().lact_swa_fwd_split(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), b, l, l, h, d, *[h * d, h * d * l] * 4, window,
                                       d ** -0.5, None, lse.data_ptr(), None, scratch.data_ptr() if cut else None, need.value,
                                       status.data_ptr(), L.stream_ptr()), "swa")
    torch.cuda.synchronize()
    assert bool((o == 7).all()) and bool((lse == 7).all())


def _address(nbytes, off, fill):
    """A buffer and the first address in it that lies `off` bytes behind a multiple of 256."""
    buf = torch.full((nbytes + 512,), fill, dtype=torch.uint8, device="cuda")
    return buf, (buf.data_ptr() + 255) // 256 * 256 + off


# scratch and outputs as they are promised to be taken: on 16 bytes
@pytest.mark.parametrize("d,l,lk,h", [(128, 1560, 4680, 12), (64, 1300, 4500, 30)])
@pytest.mark.parametrize("off", [16, 48])
def test_addresses_on_16_bytes(d, l, lk, h, off):
    import ctypes as C
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(l)
    rn = lambda n: torch.randn(1, n, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = rn(l), rn(lk), rn(lk)
    need, words = C.c_size_t(0), C.c_int64(0)
    L.check(L.lib().lact_swa_fwd_split_bytes(1, l, lk, h, d, -1, C.byref(need), C.byref(words)), "split_bytes")
    assert need.value > 0 and words.value == 0   # pairs, the last ones cut
    counters = torch.zeros(64, dtype=torch.int32, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    got = []
    for so, oo in ((0, 0), (off, 0), (0, off), (off, off)):
        scratch, at = _address(need.value, so, 0xFF)
        out, to = _address(l * h * d * 2, oo, 7)
        L.check(L.lib().lact_swa_fwd_split(q.data_ptr(), k.data_ptr(), v.data_ptr(), to, 1, l, lk, h, d, *[h * d, h * d * l],
                                           *[h * d, h * d * lk] * 2, h * d, h * d * l, -1, d ** -0.5, None, None, counters.data_ptr(), at,
                                           need.value, status.data_ptr(), L.stream_ptr()), "swa")
        torch.cuda.synchronize()
        first = to - out.data_ptr()
        assert bool((out[:first] == 7).all()) and bool((out[first + l * h * d * 2:] == 7).all())
        end = at - scratch.data_ptr() + need.value
        assert bool((scratch[:at - scratch.data_ptr()] == 0xFF).all()) and bool((scratch[end:] == 0xFF).all())
        got.append(out[first:first + l * h * d * 2].view(torch.bfloat16).view(1, l, h, d).clone())
    assert int(status[0]) == 0
    assert all(torch.equal(x, got[0]) for x in got[1:])
    want, _ = _reference(q, k, v, -1)
    # probabilities and results are rounded to bf16 (2^-9 each)
    assert float((got[0].double() - want).norm() / want.norm()) <= 6e-3


@pytest.mark.parametrize("l,lk,h,d", [(1560, 4680, 12, 128), (1300, 4500, 30, 64)])
@pytest.mark.parametrize("scratch,counters", [(True, False), (False, True), (False, False)])
def test_scratch_or_counters_alone_cut_nothing(l, lk, h, d, scratch, counters):
    """Either of them NULL: the call does without both, whatever size is given for the scratch."""
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(l)
    rn = lambda n: torch.randn(1, n, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = rn(l), rn(lk), rn(lk)
    o, buf, words = torch.empty_like(q), torch.full((256,), 0xFF, dtype=torch.uint8, device="cuda"), torch.full((64,), 3, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    L.check(L.lib().lact_swa_fwd_split(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), 1, l, lk, h, d, h * d, h * d * l,
                                       *[h * d, h * d * lk] * 2, h * d, h * d * l, -1, d ** -0.5, None, None,
                                       words.data_ptr() if counters else None, buf.data_ptr() if scratch else None, 0, status.data_ptr(),
                                       L.stream_ptr()), "swa")
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and bool((buf == 0xFF).all()) and bool((words == 3).all())
    assert torch.equal(o, _run(L, q, k, v, -1, False)[0])


# many items of uneven length, more than eight rounds of them and fewer, few items: the way that is the faster one (both measured)
@pytest.mark.parametrize("b,l,h,d,window,way", [(4, 8192, 12, 128, None, "pairs"), (16, 2048, 12, 128, 2048, "pairs"), (16, 2048, 12, 64, None, "pairs"),
                                                (8, 4096, 12, 128, 3000, "pairs"), (2, 2048, 12, 128, 256, "pairs"), (40, 200, 12, 128, None, "pairs"),
                                                (1, 3626, 12, 128, 1024, "pairs"), (1, 8192, 8, 128, None, "pairs"),
                                                (1, 2305, 8, 128, 2048, "single"), (1, 1024, 12, 128, 256, "single"), (1, 8192, 4, 128, None, "single")])
def test_the_faster_way(b, l, h, d, window, way):
    from lact_b200 import layer_ops as lo
    q, k, v = (torch.randn(b, l, h, d, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    with torch.no_grad():
        assert _kernels(lambda: lo.sliding_window_attention(q, k, v, window)) == {way}


PAIRS = {"pairs"}
CUT = {"pairs", "combine"}


# which kernel the calls of this file are compared on.  Uncut: every remainder of a pair at which its second tile or a tile's last rows are
# missing; block attention; packed sequences.  Cut: the last items of a causal launch and of block attention, all items, with and without sequences
@pytest.mark.parametrize("b,l,lk,h,d,window,cuts,way", [
    *[(1, l, l, 300, d, w, (), PAIRS) for d in (64, 128) for l, w in ((1, 0), (127, 40), (128, 128), (129, 1), (255, 0), (256, 128), (257, 129),
                                                                     (385, 256), (511, 130), (513, 600))],
    *[(1, l, 700, 148, 128, -1, (), PAIRS) for l in (129, 255, 257)], (1, 300, 1025, 148, 64, -1, (), PAIRS),
    (1, 1100, 1100, 40, 128, 0, (), PAIRS), (1, 257, 257, 74, 64, 200, (), PAIRS), (3, 130, 127, 30, 64, -1, (), PAIRS),
    (1, 900, 900, 100, 64, 0, (), PAIRS), (1, 1100, 1100, 60, 128, 300, (255, 257, 1000), PAIRS), (1, 300, 300, 200, 128, 0, (), PAIRS),
    (1, 2600, 2500, 14, 128, -1, (), CUT), (2, 1900, 2600, 10, 64, -1, (), CUT), (1, 5000, 5000, 2, 128, 0, (), CUT),
    (1, 5000, 5000, 2, 128, 0, (1, 2, 383, 4999), CUT), (1, 5000, 5000, 2, 64, 0, (128, 1000, 3073), CUT), (1, 7000, 7000, 2, 64, 5600, (), CUT)])
def test_the_kernel_that_is_compared(b, l, lk, h, d, window, cuts, way):
    g = torch.Generator(device="cuda").manual_seed(l + h + d)
    rn = lambda n: torch.randn(b, n, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = rn(l), rn(lk), rn(lk)
    starts = None
    if cuts:
        starts = torch.zeros(l, dtype=torch.int32, device="cuda")
        for c in cuts:
            starts[c:] = c
    _compare(q, k, v, window, way == CUT, starts)
    assert _kernels(_prepared(q, k, v, window, way == CUT, starts)[0]) == way


# keys in two runs on pairs that are cut over both: the first ends on a tile's end, just past one, inside one
@pytest.mark.parametrize("cached", [3120, 3072, 3073, 2999])
@pytest.mark.parametrize("l,new,h,d", [(1560, 1560, 12, 128), (1300, 1400, 30, 64)])
def test_cut_over_a_cache_and_new_keys(l, cached, new, h, d):
    from lact_b200 import layer_ops as lo
    g = torch.Generator(device="cuda").manual_seed(cached)
    rn = lambda *s: torch.randn(*s, h, d, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v, cache = rn(1, l), rn(1, new), rn(1, new), rn(2, cached)
    call = lambda: lo.sliding_window_attention_inference(q, k, v, new, kv_cache=cache)
    o = call()
    assert _kernels(call) == CUT
    want, _ = _reference(q, torch.cat([cache[:1], k], 1), torch.cat([cache[1:], v], 1), -1)
    # probabilities and results are rounded to bf16 (2^-9 each)
    assert float((o.double() - want).norm() / want.norm()) <= 6e-3


@pytest.mark.parametrize("l,lk,h,window,way", [(300, 300, 200, 0, PAIRS), (1560, 4680, 12, -1, CUT), (5000, 5000, 2, 0, CUT)])
def test_pairs_after_an_earlier_failure(l, lk, h, window, way):
    """Outputs and the status word stay what they were."""
    rn = lambda n: torch.randn(1, n, h, 128, device="cuda").to(torch.bfloat16)
    call, o, lse, status = _prepared(rn(l), rn(lk), rn(lk), window, way == CUT, failed=True)
    assert _kernels(call) == way
    assert bool((o == 7).all()) and bool((lse == 7).all()) and int(status[0]) == 101


# small calls, where a launch of pairs costs more than its rounds save; a launch of uneven items that single tiles cut; and others like them that pairs are
# faster at (all measured both ways)
@pytest.mark.parametrize("b,l,lk,h,d,window,way", [
    (1, 121, 121, 24, 64, 0, "single"), (3, 128, 128, 16, 64, 12, "single"), (2, 239, 239, 3, 64, 0, "single"), (1, 128, 128, 4, 64, 64, "single"),
    (1, 768, 132, 24, 128, -1, "single"), (1, 4736, 249, 1, 128, -1, "single"), (1, 648, 2912, 24, 64, -1, "single"), (1, 738, 738, 6, 64, 14, "single"),
    (1, 6234, 6234, 3, 64, 5610, "single"), (1, 8192, 8192, 4, 128, 0, "single"),
    (4, 5632, 96, 24, 64, -1, "pairs"), (8, 1485, 1485, 32, 128, 29, "pairs"), (3, 130, 127, 30, 64, -1, "pairs"), (1, 257, 257, 74, 64, 200, "pairs")])
def test_the_faster_way_of_small_and_of_cut_calls(b, l, lk, h, d, window, way):
    rn = lambda n: torch.randn(b, n, h, d, device="cuda").to(torch.bfloat16)
    assert _kernels(_prepared(rn(l), rn(lk), rn(lk), window, True)[0]) == {way}
