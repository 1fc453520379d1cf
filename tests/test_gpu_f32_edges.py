"""fp32 mode at the edges of what it takes."""
import pytest
import torch

from test_gpu_overlapping_ranges import fill_free_memory

pytestmark = pytest.mark.gpu
NAMES = ("w0", "w1", "w2", "q", "k", "v", "lr0", "lr1", "lr2")


def _inputs(B, L, D, H, seed=1):
    from oracle import lact_oracle as orc
    return {n: t.cuda() for n, t in orc.make_inputs(B, L, D, H, seed=seed).items()}


def _close(a, b, tol):
    assert torch.isfinite(a).all()
    assert float((a - b).abs().max()) <= tol * float(b.abs().max())


def test_momentum_after_an_empty_first_update():
    import lact_b200 as lb
    from lact_b200 import ops
    from lact_b200 import program as P
    L, n = 96, 48
    i = _inputs(2, L, 32, 16)
    args = [i[x] for x in NAMES]
    steps = [(P.APPLY, 0, n, 0), (P.UPDATE, 0, n, 0), (P.APPLY, n, L, n), (P.UPDATE, n, L, 0)]
    want = ops.scan(*args, steps, momentum=i["momentum"], return_state=True, return_momentum=True)
    for empty in (1, 2):
        fill_free_memory()
        got = ops.scan(*args, [(P.UPDATE, 0, 0, 0)] * empty + steps, momentum=i["momentum"], return_state=True, return_momentum=True)
        got_o = ops.scan(*args, [(P.UPDATE, 0, 0, 0)] * empty + steps, momentum=i["momentum"], return_state=True)
        lb.synchronize_and_check()
        for a, b in zip(list(got) + list(got_o), list(want) + list(want[:4])):
            assert torch.equal(a, b)


@pytest.mark.parametrize("B,L", [(1100, 9), (1025, 150)])
def test_many_entries(B, L):
    import lact_b200 as lb
    i = _inputs(B, L, 4, 8)
    chunk = 4 if L < 100 else 149
    run = lambda s, e: lb.block_causal_lact_swiglu(*[i[n][s:e] for n in NAMES], chunk_size=chunk, momentum=i["momentum"][s:e])
    got = run(0, B)
    _close(got, torch.cat([run(0, 513), run(513, B)]), 1e-5)   # fp32 sums of at most 149 terms, split differently


@pytest.mark.parametrize("D,H", [(1036, 8), (16, 1048)])
def test_rows_longer_than_an_update_takes(D, H):
    import lact_b200 as lb
    i = _inputs(1, 20, D, H)
    got = lb.block_causal_lact_swiglu(*[i[n] for n in NAMES], chunk_size=32)   # one chunk: no update
    w0, w1, w2, q = (i[n].double() for n in ("w0", "w1", "w2", "q"))
    want = (torch.nn.functional.silu(q @ w0.transpose(1, 2)) * (q @ w2.transpose(1, 2))) @ w1.transpose(1, 2)
    _close(got.double(), want, 1e-5)
    with pytest.raises(ValueError):
        lb.block_causal_lact_swiglu(*[i[n] for n in NAMES], chunk_size=8)


def test_bf16_gate_is_averaged_in_fp32():
    import lact_b200 as lb
    i = _inputs(2, 90, 32, 16)
    gate = i["momentum"].to(torch.bfloat16)
    run = lambda m: lb.block_causal_lact_swiglu(*[i[n] for n in NAMES], chunk_size=30, momentum=m)
    assert torch.equal(run(gate), run(gate.float()))


@pytest.mark.parametrize("M,N,K", [(3, 4, 5), (130, 64, 17), (65, 72, 16)])
@pytest.mark.parametrize("shift", [(0, 0, 1), (1, 0, 0), (1, 3, 2)])
def test_product_of_arrays_off_sixteen_bytes(M, N, K, shift):
    """lact_sgemm_f32 takes arrays that start on any element."""
    from lact_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(M)
    at = lambda n, s: torch.randn(n + s, device="cuda", generator=g)[s:]
    a, b, c = at(2 * M * K, shift[0]), at(2 * N * K, shift[1]), at(2 * M * N, shift[2])
    want = a.view(2, M, K).double() @ b.view(2, N, K).double().transpose(1, 2) + c.view(2, M, N).double()
    L.check(L.lib().lact_sgemm_f32(a.data_ptr(), 0, b.data_ptr(), 0, c.data_ptr(), 1, None, 2, M, N, K, L.stream_ptr()), "sgemm")
    torch.cuda.synchronize()
    _close(c.view(2, M, N).double(), want, 1e-5)   # fp32 sums of at most 18 terms
