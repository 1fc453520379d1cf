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
