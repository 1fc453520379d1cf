"""Device status and stream capture."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = """
import ctypes as C, torch
import lact_b200 as lb
from lact_b200 import _lib as L
from lact_b200 import layer_ops as lo
g = torch.Generator(device="cuda").manual_seed(0)
rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
bf = lambda *s: rn(*s).to(torch.bfloat16)
def scan_args(B=1, n=256, D=64, H=64):
    unit = lambda t: (t / t.norm(dim=-1, keepdim=True)).to(torch.bfloat16)
    return [rn(B, H, D) / 8, rn(B, D, H) / 8, rn(B, H, D) / 8, unit(rn(B, n, D)), unit(rn(B, n, D)), bf(B, n, D)] + [torch.rand(B, n, 1, device="cuda") / 8 for _ in range(3)]
def train(leaves, dout):
    o = lb.block_causal_lact_swiglu(*leaves, chunk_size=64, use_muon=True)
    return [o.detach()] + list(torch.autograd.grad(o, leaves, dout))
def make(kind):
    if kind == "attention":
        t = [bf(1, 300, 2, 64) for _ in range(3)]
        return lambda: [lo.sliding_window_attention(*t, 128)]
    if kind == "ffn":
        t = bf(2, 128, 64) / 8, bf(2, 64, 64) / 8, bf(2, 40, 64)
        return lambda: [lb.fused_swiglu_ffn_fwd(*t)]
    if kind == "train":
        leaves, dout = [t.requires_grad_(True) for t in scan_args()], bf(1, 256, 64)
        return lambda: train(leaves, dout)
    if kind == "newton_schulz":
        t = rn(2, 64, 128)
        return lambda: [lb.zeropower_via_newtonschulz5(t)]
    t = scan_args()
    return lambda: [lb.block_causal_lact_swiglu(*t, chunk_size=64, use_muon=True)]
"""


def _python(code, **env):
    r = subprocess.run([sys.executable, "-c", SETUP + code], cwd=ROOT, capture_output=True, text=True, timeout=300, env={**os.environ, **env})
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.parametrize("kind", ["attention", "ffn", "train"])
def test_graphs_of_one_stream_replay_in_any_order(kind):
    ns = {}
    exec(SETUP + f"\ncall = make({kind!r})", ns)
    call, lb = ns["call"], ns["lb"]
    want = call()
    lb.synchronize_and_check()
    stream, pool = torch.cuda.Stream(), torch.cuda.graph_pool_handle()
    filler, first, second = (torch.cuda.CUDAGraph() for _ in range(3))
    with torch.cuda.graph(filler, pool=pool, stream=stream):   # leaves non-zero words in the pool's memory
        junk = [torch.full((n,), 1, dtype=torch.int32, device="cuda") for n in (1 << 20, 1 << 16, 1 << 12, 128) for _ in range(24)]
        del junk
    filler.replay()
    torch.cuda.synchronize()
    with torch.cuda.graph(first, pool=pool, stream=stream):
        out1 = call()
    with torch.cuda.graph(second, pool=pool, stream=stream):
        out2 = call()
    for graph, out in ((second, out2), (first, out1), (second, out2)):
        filler.replay()
        for t in out:
            t.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(out, want):
            assert torch.equal(a, b)
    again = call()   # and eager calls after them
    lb.synchronize_and_check()
    for a, b in zip(again, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("kind", ["attention", "ffn", "train", "scan", "newton_schulz"])
def test_first_call_of_a_process_inside_a_capture(kind):
    _python(f"""
call = make({kind!r})
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out = call()
graph.replay()
torch.cuda.synchronize()
want = call()
lb.synchronize_and_check()
assert all(torch.equal(a, b) for a, b in zip(out, want))
""")


def test_failure_in_a_process_that_calls_no_registered_operator():
    _python("""
lb.zeropower_via_newtonschulz5(rn(1, 64, 64))
dev = torch.device("cuda", 0)
ws = L.workspace(1 << 20, dev)
ws[:256].zero_()
L.check(L.lib().lact_set_wait_limit_ns(1_000_000), "limit")
L.check(L.lib().lact_debug_wait_timeout(ws.data_ptr(), L.stream_ptr()), "timeout")
torch.cuda.synchronize()
try:
    L.mark_pending(ws)
    lb.synchronize_and_check()
except lb.LactError:
    pass
else:
    raise SystemExit("not reported")
lb.zeropower_via_newtonschulz5(rn(1, 64, 64))
lb.synchronize_and_check()
""")


def _fail_on_host():
    from lact_b200 import _lib as L
    word = C.POINTER(C.c_int32)()
    L.check(L.lib().lact_status_host_word(C.byref(word)), "word")
    word[0] = 101


@pytest.mark.parametrize("kind", ["scan", "attention", "ffn", "grads"])
def test_failure_found_in_a_backward_is_a_lact_error(kind):
    ns = {}
    exec(SETUP, ns)
    lb, lo, bf, rn = (ns[n] for n in ("lb", "lo", "bf", "rn"))
    leaf = lambda t: t.requires_grad_(True)
    if kind == "scan":
        o = lb.block_causal_lact_swiglu(*[leaf(t) for t in ns["scan_args"]()], chunk_size=64)
    elif kind == "attention":
        o = lo.sliding_window_attention(*[leaf(bf(1, 300, 2, 64)) for _ in range(3)], 128)
    elif kind == "ffn":
        o = lb.fused_swiglu_ffn_fwd(leaf(bf(2, 128, 64)), leaf(bf(2, 64, 64)), leaf(bf(2, 40, 64)))
    else:
        o = lb.fused_lact_swiglu_ffn_fast_weight_grads(leaf(bf(2, 128, 64)), leaf(bf(2, 64, 64)), leaf(bf(2, 40, 64)), leaf(bf(2, 40, 64)),
                                                       *[torch.rand(2, 40, device="cuda") for _ in range(3)])[0]
    lb.synchronize_and_check()
    _fail_on_host()
    with pytest.raises(lb.LactError, match="101"):
        o.backward(torch.ones_like(o))
    with pytest.raises(ValueError):   # (arguments stay ValueError)
        lb.block_causal_lact_swiglu(*ns["scan_args"]()[:8], torch.rand(1, 3, 1, device="cuda"), chunk_size=64)
    _fail_on_host()
    with pytest.raises(lb.LactError, match="101"):
        lb.block_causal_lact_swiglu(*ns["scan_args"](), chunk_size=64)


def test_sync_check_covers_backwards():
    out = _python("""
leaves, dout = [t.requires_grad_(True) for t in scan_args()], bf(1, 256, 64)
o = lb.block_causal_lact_swiglu(*leaves, chunk_size=64)
torch.cuda.set_sync_debug_mode("error")
try:
    torch.autograd.grad(o, leaves, dout)
except RuntimeError as e:
    print("waited" if "synchronizing" in str(e) else e)
torch.cuda.set_sync_debug_mode("default")
# and a capture is left alone
call = make("train")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    call()
""", LACT_B200_SYNC_CHECK="1")
    assert "waited" in out
