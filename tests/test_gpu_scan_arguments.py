"""Arguments of the recurrence that reach past its usual form."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
NAMES = ("w0", "w1", "w2", "q", "k", "v", "lr0", "lr1", "lr2")


def _inputs(B, L, D, H, act=BF16, seed=2):
    from oracle import lact_oracle as orc
    return {n: t.cuda() for n, t in orc.make_inputs(B, L, D, H, seed=seed, act_dtype=act).items()}


@pytest.mark.parametrize("act,train", [(BF16, False), (BF16, True), (torch.float32, False)])
def test_tensors_off_the_device_are_refused(act, train):
    """Refused on the host, before anything is enqueued: every tensor argument in turn on the CPU."""
    from lact_b200 import ops
    from lact_b200 import program as P
    i = _inputs(1, 64, 32, 32, act)
    m_init = [torch.zeros_like(i[n]) for n in ("w0", "w1", "w2")]
    if train:
        i["w0"].requires_grad_(True)
    for name in NAMES + ("momentum",) + (() if train else ("m0", "m1", "m2")):
        a, m = dict(i), None if train else list(m_init)
        if name in a:
            a[name] = a[name].detach().cpu()
        else:
            m[int(name[1])] = m[int(name[1])].cpu()
        if name != "w0":
            a["w0"] = i["w0"]
        with pytest.raises((RuntimeError, ValueError), match="CUDA tensors only|same device"):
            ops.scan(*[a[n] for n in NAMES], P.causal_program(64, 32), momentum=a["momentum"], m_init=m)


@pytest.mark.parametrize("which", [("w0",), ("w1",), ("w2",), ("w1", "w2")])
def test_c_abi_returns_each_weight_by_itself(which):
    """The final weights are optional one by one (each out pointer may be NULL)."""
    from lact_b200 import _lib as L
    from lact_b200 import ops
    from lact_b200 import program as P
    B, n, D, H = 2, 128, 64, 32
    i = _inputs(B, n, D, H)
    steps = P.causal_program(n, 64)
    want = dict(zip(("o", "w0", "w1", "w2"), ops.scan(*[i[x] for x in NAMES], steps, return_state=True)))
    cfg, io = L.ScanConfig(), L.ScanIO()
    cfg.B, cfg.L, cfg.D, cfg.H, cfg.out_len, cfg.act_dtype, cfg.renorm, cfg.w_scale = B, n, D, H, n, L.LACT_BF16, L.RENORM_EPS_OUTSIDE, 1.0
    for x in ("q", "k", "v", "o"):
        setattr(cfg, x + "_bs", n * D)
        setattr(cfg, x + "_ts", D)
    out = {x: torch.full(want[x].shape, float("nan"), device="cuda") for x in which}
    o = torch.empty(B, n, D, dtype=BF16, device="cuda")
    for x in NAMES:
        setattr(io, x, i[x].data_ptr())
    io.o = o.data_ptr()
    for x in which:
        setattr(io, x + "_out", out[x].data_ptr())
    m = len(steps)
    kind, start, end, outs = ((t * m)(*[s[j] for s in steps]) for j, t in enumerate((C.c_int32, C.c_int64, C.c_int64, C.c_int64)))
    need = C.c_size_t(0)
    L.check(L.lib().lact_scan_workspace_bytes(C.byref(cfg), m, kind, start, end, C.byref(need)), "bytes")
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    L.check(L.lib().lact_scan_fwd(C.byref(cfg), C.byref(io), m, kind, start, end, outs, ws.data_ptr(), need, L.stream_ptr()), "scan")
    torch.cuda.synchronize()
    assert torch.equal(o, want["o"])
    for x in which:
        assert torch.equal(out[x], want[x]), x


@pytest.mark.parametrize("offset", [0, 2, 4])
def test_state_arrays_on_any_byte(offset):
    """Momentum in and out and the final weights may start anywhere (they are copied, byte by byte if need be)."""
    from lact_b200 import _lib as L
    from lact_b200 import ops
    from lact_b200 import program as P
    B, n, D, H = 2, 64, 64, 32
    i = _inputs(B, n, D, H)
    g = torch.Generator(device="cuda").manual_seed(1)
    m = [torch.randn(i[w].shape, device="cuda", generator=g) for w in ("w0", "w1", "w2")]
    gate = i["momentum"].float().contiguous()
    steps = [(P.UPDATE, 0, n, 0), (P.APPLY, 0, n, 0)]
    want = ops.scan(*[i[x] for x in NAMES], steps, momentum=gate, m_init=m, return_state=True, return_momentum=True)
    cfg, io = L.ScanConfig(), L.ScanIO()
    cfg.B, cfg.L, cfg.D, cfg.H, cfg.out_len, cfg.act_dtype, cfg.renorm, cfg.w_scale = B, n, D, H, n, L.LACT_BF16, L.RENORM_EPS_OUTSIDE, 1.0
    cfg.use_momentum = 1
    for x in ("q", "k", "v", "o"):
        setattr(cfg, x + "_bs", n * D)
        setattr(cfg, x + "_ts", D)
    for x in NAMES:
        setattr(io, x, i[x].data_ptr())
    o = torch.empty(B, n, D, dtype=BF16, device="cuda")
    io.o, io.momentum = o.data_ptr(), gate.data_ptr()
    size = B * H * D * 4
    packed = {x: torch.zeros(size + 16, dtype=torch.uint8, device="cuda") for x in ("m0_in", "m1_in", "m2_in", "w0_out", "w1_out", "w2_out",
                                                                                   "m0_out", "m1_out", "m2_out")}
    for x, t in zip(("m0_in", "m1_in", "m2_in"), m):
        packed[x][offset:offset + size] = t.reshape(-1).view(torch.uint8)
    for x, t in packed.items():
        setattr(io, x, t.data_ptr() + offset)
    kind, start, end, outs = ((t * 2)(*[s[j] for s in steps]) for j, t in enumerate((C.c_int32, C.c_int64, C.c_int64, C.c_int64)))
    need = C.c_size_t(0)
    L.check(L.lib().lact_scan_workspace_bytes(C.byref(cfg), 2, kind, start, end, C.byref(need)), "bytes")
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    L.check(L.lib().lact_scan_fwd(C.byref(cfg), C.byref(io), 2, kind, start, end, outs, ws.data_ptr(), need, L.stream_ptr()), "scan")
    torch.cuda.synchronize()
    assert torch.equal(o, want[0])
    for x, t in zip(("w0_out", "w1_out", "w2_out", "m0_out", "m1_out", "m2_out"), want[1:]):
        assert torch.equal(packed[x][offset:offset + size].clone().view(torch.float32).view(t.shape), t), x


@pytest.mark.parametrize("act", [BF16, torch.float32])
@pytest.mark.parametrize("muon", [False, True])
def test_nan_gate_of_the_first_chunk_reaches_the_weights(act, muon):
    import lact_b200 as lb
    i = _inputs(2, 256, 64, 64, act)
    clean = lb.block_causal_lact_swiglu(*[i[n] for n in NAMES], chunk_size=64, use_muon=muon, momentum=i["momentum"])
    for bad in (float("nan"), float("inf")):
        m = i["momentum"].clone()
        m[1, 3] = bad
        o = lb.block_causal_lact_swiglu(*[i[n] for n in NAMES], chunk_size=64, use_muon=muon, momentum=m)
        lb.synchronize_and_check()
        assert torch.equal(o[0], clean[0]) and torch.equal(o[1, :64], clean[1, :64])
        assert bool(o[1, 64:].isnan().all())   # bad * 0 (the state before the first update)


def test_gate_gradient_over_many_updates_is_summed_in_fp32():
    from lact_b200 import ops
    from lact_b200 import program as P
    i = _inputs(2, 64, 32, 32)
    steps = [(P.UPDATE, 0, 32, 0)] * 150 + [(P.APPLY, 0, 64, 0)]
    dO = torch.randn(2, 64, 32, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).to(BF16)

    def grad(m):
        m = m.requires_grad_(True)
        return torch.autograd.grad(ops.scan(*[i[n] for n in NAMES], steps, momentum=m), m, dO)[0]
    gate = torch.full((2, 64, 1), 0.5, device="cuda")   # its mean is exact in bf16
    a, b = grad(gate.to(BF16)), grad(gate)
    assert a.dtype == BF16 and float(b.abs().max()) > 0
    assert torch.equal(a, b.to(BF16))
