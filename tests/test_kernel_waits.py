"""Hand-overs between the warps of a kernel, walked through on the CPU: a wait by parity holds for one phase of a barrier, so no
barrier may complete a second phase before the waiting warp has looked at the first."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lact_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


class _Barrier:
    def __init__(self):
        self.phases = 0   # completed

    def passes(self, parity):   # what mbarrier.try_wait.parity answers
        return (self.phases & 1) != parity


def _all_end(agents, slowest):
    """Runs the agents (generators of the waits they come to) with `slowest` taking a step only when no other can; True if all end."""
    at = {a: next(g, None) for a, g in agents.items()}

    def step(a):
        ready = at[a] is not None and at[a][0].passes(at[a][1])
        if ready:
            at[a] = next(agents[a], None)
        return ready

    while True:
        if not any([step(a) for a in agents if a != slowest]) and not step(slowest):
            return all(w is None for w in at.values())


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7, 20])
@pytest.mark.parametrize("slowest", ["values", "softmax", "products"])
def test_per_query_values_of_the_attention_backward(tiles, slowest):
    """Mode 0 of the attention backward: one warp stages the values of a tile, the softmax warps use them, a third issues the
    products.  The wait before a stage is written again is the one in the source."""
    m = re.search(r"if \(t >= 2 && !mbar_wait_warp\((&?)(st_empty|ds_full)(\[t & 1\])?, (.+?), abort_flag\)\) \{[^}]*\}\s*// .*tile t - 2",
                  _source("swa_bwd.cuh"))
    assert m is not None
    barrier, per_stage, parity = m.group(2), m.group(3) is not None, m.group(4)
    bar = {n: [_Barrier(), _Barrier()] for n in ("st_full", "st_empty")} | {n: _Barrier() for n in ("s_full", "dp_full", "p_full", "ds_full")}

    def values():
        for t in range(tiles):
            if t >= 2:
                yield (bar[barrier][t & 1] if per_stage else bar[barrier]), eval(parity, {"t": t})
            bar["st_full"][t & 1].phases += 1

    def softmax():
        for t in range(tiles):
            yield bar["st_full"][t & 1], (t >> 1) & 1
            yield bar["s_full"], t & 1
            bar["p_full"].phases += 1
            yield bar["dp_full"], t & 1
            bar["ds_full"].phases += 1
            bar["st_empty"][t & 1].phases += 1

    def products():
        bar["s_full"].phases += 1
        bar["dp_full"].phases += 1
        for t in range(tiles):
            yield bar["p_full"], t & 1
            if t + 1 < tiles:
                bar["s_full"].phases += 1
            yield bar["ds_full"], t & 1
            if t + 1 < tiles:
                bar["dp_full"].phases += 1

    agents = {"values": values(), "softmax": softmax(), "products": products()}
    assert _all_end(agents, slowest)


@pytest.mark.parametrize("name", ["umma_gemm.cuh", "pair_gemm.cuh", "ns_fused.cuh", "ns_bwd_fused.cuh", "ns_chip.cuh"])
def test_whether_to_take_part_is_decided_once_per_cta(name):
    """The warps of these kernels meet at named barriers, which have no time limit, if they take part: no thread may decide that
    from its own reading of the status word.  (A thread that reports a failure of its own may look at it, or one that tells all.)"""
    reads = [line for line in _source(name).splitlines() if ".status) == kStatusOk" in line or ".status) != kStatusOk" in line]
    assert all(any(w in line for w in ("failed &&", "if (threadIdx.x == 0)", "__syncthreads_or(")) for line in reads), reads
    assert reads or "earlier_launch_failed(args.status)" in _source(name)


def test_the_epilogue_warps_decide_at_a_barrier():
    body = re.search(r"bool earlier_launch_failed\(.*?\n}", _source("umma_gemm.cuh"), re.S).group(0)
    assert "if (uniform_warp_index() >= 2) set = named_barrier_any(" in body


def test_a_warp_meets_again_before_aligned_loads_of_tensor_memory():
    """Attention on pairs: the log-sum-exp is stored by the rows below the end alone, the loads behind it want the whole warp."""
    between = re.search(r"inv = finish_row\(\);(.*?)own\(c, v\);", _source("swa_pairs.cuh"), re.S).group(1)
    assert "__syncwarp();" in between


class _Counted(_Barrier):
    def __init__(self, count):
        super().__init__()
        self.count, self.arrived = count, 0

    def arrive(self, n=1):
        self.arrived += n
        assert self.arrived <= self.count
        if self.arrived == self.count:
            self.phases, self.arrived = self.phases + 1, 0


def test_the_one_launch_gradient_meets_at_its_named_barrier_by_one_decision():
    """Its epilogue warps meet at a named barrier; the second issuing warp, which does not, reads the status word by itself."""
    text = _source("grad_fused.cuh")
    reads = [line for line in text.splitlines() if ".status))" in line and "kStatusOk" in line]
    assert len(reads) == 1 and re.search(r"failed = warp < 2 \+ kEpiWarps \? earlier_launch_failed\(a\.status\)\s*:", text)


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 6, 7, 12, 13])
@pytest.mark.parametrize("slowest", ["load", "first", "second", "warp0", "warp1"])
def test_rings_of_the_one_launch_gradient(tiles, slowest):
    """The fast-weight gradient in one launch: rings of three (k) and two (v), two buffers of first products, one set of planes."""
    one = lambda: _Counted(1)
    k_full, k_empty, v_full, v_empty = [one() for _ in range(3)], [one() for _ in range(3)], [one(), one()], [one(), one()]
    y_full, y_empty = [one(), one()], [_Counted(2), _Counted(2)]
    w_full, planes_full, planes_empty, acc_full = one(), _Counted(2), one(), one()
    k, v, y, planes, done = [None] * 3, [None] * 2, [None] * 2, [None, None], []

    def load():
        k[0], v[0] = 0, 0
        k_full[0].arrive(), w_full.arrive(), v_full[0].arrive()
        ks, kph = 1, 1
        for i in range(1, tiles):
            yield k_empty[ks], kph
            assert k[ks] is None or k[ks] in done
            k[ks] = i
            k_full[ks].arrive()
            ks, kph = (0, kph ^ 1) if ks == 2 else (ks + 1, kph)
            yield v_empty[i & 1], ((i >> 1) & 1) ^ 1
            assert v[i & 1] is None or v[i & 1] in done
            v[i & 1] = i
            v_full[i & 1].arrive()

    def first():
        ks, kph = 0, 0
        yield w_full, 0
        for i in range(tiles):
            s, ph = i & 1, (i >> 1) & 1
            yield y_empty[s], ph ^ 1
            yield k_full[ks], kph
            assert k[ks] == i
            ks, kph = (0, kph ^ 1) if ks == 2 else (ks + 1, kph)
            yield v_full[s], ph
            assert v[s] == i
            y[s] = i
            y_full[s].arrive()

    def epilogue(warp):
        for i in range(tiles):
            s, ph = i & 1, (i >> 1) & 1
            yield y_full[s], ph
            assert y[s] == i
            y_empty[s].arrive()
            if i > 0:
                yield planes_empty, (i - 1) & 1
            assert i == 0 or i - 1 in done
            planes[warp] = i
            planes_full.arrive()
        yield acc_full, 0
        assert done == list(range(tiles))

    def second():
        ks = 0
        for i in range(tiles):
            yield planes_full, i & 1
            assert planes == [i, i] and k[ks] == i and v[i & 1] == i
            done.append(i)
            v_empty[i & 1].arrive(), k_empty[ks].arrive(), planes_empty.arrive()
            ks = 0 if ks == 2 else ks + 1
        acc_full.arrive()

    assert _all_end({"load": load(), "first": first(), "second": second(), "warp0": epilogue(0), "warp1": epilogue(1)}, slowest)


# (key tiles of group 0, of group 1) of a CTA's items in turn: equal ones, a diagonal, a band, pieces in which a group has none or both have none,
# a last pair without a second tile (None)
@pytest.mark.parametrize("items", [[((0, 1), (0, 1))], [((0, 5), (0, 5))] * 3, [((0, 1), (0, 2)), ((0, 3), (0, 4)), ((2, 7), (3, 8))],
                                   [((0, 4), (4, 4)), ((4, 4), (4, 6)), ((6, 6), (6, 6)), ((1, 3), (1, 4))], [((2, 9), None), ((0, 1), None), ((0, 2), (0, 2))],
                                   [((3, 3), (3, 3))], [((0, 2), (1, 3))] * 4])
@pytest.mark.parametrize("slowest", ["load", "products0", "products1", "softmax0", "softmax1", "correction"])
def test_rings_of_the_attention_on_pairs(items, slowest):
    """Rings of two for keys and values run on across items; groups begin and end on tiles of their own."""
    one = lambda: [_Counted(1), _Counted(1)]
    q_full, q_empty, k_full, v_full, s_full, o_full, o_empty, a_full, ml_full, p_full = (one() for _ in range(10))
    k_empty, v_empty, p_half = ([_Counted(2), _Counted(2)] for _ in range(3))   # both groups; softmax and correction
    none = (0, 0)
    work = [(a, b or none, min(a[0], b[0]) if b and a[0] < a[1] and b[0] < b[1] else a[0] if a[0] < a[1] or not b else b[0],
             max(a[1], (b or none)[1]), b is not None) for a, b in items]
    q, k, v = [None] * 2, [None] * 2, [None] * 2
    s, p, o, factor, ml = [None] * 2, [None] * 2, [None] * 2, [None] * 2, [None] * 2   # what lies there: (item, tile), of o the last tile in it
    rows = []

    def load():
        n, parts = 0, [0, 0]
        for i, (a, b, first, last, _) in enumerate(work):
            for t in range(first, last):
                for g, (lo, hi) in enumerate((a, b)):
                    if t == lo and t < hi:
                        parts[g] += 1
                        if parts[g] > 1:
                            yield q_empty[g], (parts[g] - 2) & 1
                        q[g] = i
                        q_full[g].arrive()
                sb, ph = n & 1, ((n >> 1) & 1) ^ 1
                yield k_empty[sb], ph
                k[sb] = (i, t)
                k_full[sb].arrive()
                yield v_empty[sb], ph
                v[sb] = (i, t)
                v_full[sb].arrive()
                n += 1

    def products(g):
        n = tiles = parts = 0
        pending = None
        flat = [(i, t, w[g]) for i, w in enumerate(work) for t in range(w[2], w[3])] + [None]
        for at in flat:
            sb, ph = n & 1, (n >> 1) & 1
            if at is not None:
                yield k_full[sb], ph
            if pending is not None:
                (pi, pt, (lo, hi)), stage, parity = pending
                yield v_full[stage], parity
                if pt == lo and parts > 1:
                    yield o_empty[g], parts & 1
                yield p_half[g], tiles & 1
                yield p_full[g], tiles & 1
                assert p[g] == (pi, pt) and v[stage] == (pi, pt)
                assert (o[g] is None or o[g][0] != pi) if pt == lo else o[g] == (pi, pt - 1, "corrected")
                o[g] = (pi, pt)
                v_empty[stage].arrive()
                if pt + 1 == hi:
                    o_full[g].arrive()
                tiles += 1
                pending = None
            if at is None:
                return
            i, t, (lo, hi) = at
            if not lo <= t < hi:
                yield v_full[sb], ph
                k_empty[sb].arrive(), v_empty[sb].arrive()
            else:
                if t == lo:
                    yield q_full[g], parts & 1
                    parts += 1
                assert q[g] == i and k[sb] == (i, t)
                s[g] = (i, t)
                s_full[g].arrive(), k_empty[sb].arrive()
                pending = (at, sb, ph)
                if t + 1 == hi:
                    q_empty[g].arrive()
            n += 1

    def softmax(g):
        tiles = parts = 0
        for i, w in enumerate(work):
            lo, hi = w[g]
            if lo >= hi:
                continue
            for t in range(lo, hi):
                yield s_full[g], tiles & 1
                tiles += 1
                assert s[g] == (i, t)
                if t > lo:
                    assert factor[g] is None
                    factor[g] = (i, t)
                    a_full[g].arrive()
                p[g] = (i, t)
                p_half[g].arrive(1 if t > lo else 2)
                p_full[g].arrive()
            if parts > 0:
                yield o_empty[g], (parts - 1) & 1
            parts += 1
            assert ml[g] is None
            ml[g] = i
            ml_full[g].arrive()

    def correction():
        tiles, parts = [0, 0], [0, 0]
        for i, (a, b, first, last, second) in enumerate(work):
            ends = [a[1] if a[0] < a[1] else last, -1 if not second else b[1] if b[0] < b[1] else last]
            for t in range(first, last + 1):
                for g, (lo, hi) in enumerate((a, b)):
                    if t != ends[g]:
                        continue
                    if lo < hi:
                        parts[g] += 1
                        yield ml_full[g], (parts[g] - 1) & 1
                        yield o_full[g], (parts[g] - 1) & 1
                        assert ml[g] == i and o[g] == (i, hi - 1)
                        ml[g] = None
                        o_empty[g].arrive()
                    rows.append((i, g))
                for g, (lo, hi) in enumerate((a, b)):
                    if lo < t < hi:
                        yield a_full[g], tiles[g] & 1
                        tiles[g] += 1
                        assert factor[g] == (i, t) and o[g] == (i, t - 1)
                        factor[g], o[g] = None, (i, t - 1, "corrected")
                        p_half[g].arrive()

    assert _all_end({"load": load(), "products0": products(0), "products1": products(1), "softmax0": softmax(0), "softmax1": softmax(1),
                     "correction": correction()}, slowest)
    assert sorted(rows) == [(i, g) for i, w in enumerate(work) for g in range(1 + w[4])]
