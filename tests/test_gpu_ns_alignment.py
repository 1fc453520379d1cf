"""Newton-Schulz of gradients that are views into a packed buffer, off the 16-byte boundary its kernels read from."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one matrix per SM, and matrices too large for that
@pytest.mark.parametrize("shape", [(3, 64, 128), (2, 192, 128), (2, 256, 384)])
@pytest.mark.parametrize("dtype,shift", [(torch.bfloat16, 4), (torch.bfloat16, 1), (torch.float32, 1), (torch.float32, 2)])
def test_views_off_sixteen_bytes(shape, dtype, shift):
    import lact_b200 as lb
    n = shape[0] * shape[1] * shape[2]
    gen = torch.Generator(device="cuda").manual_seed(n + shift)
    view = torch.randn(n + shift, device="cuda", generator=gen).to(dtype)[shift:].view(shape)
    assert view.is_contiguous() and view.data_ptr() % 16
    d = torch.randn(shape, device="cuda", generator=gen).to(torch.bfloat16)
    leaf, plain = view.detach().requires_grad_(True), view.clone().requires_grad_(True)
    for steps in (None, 3):
        assert torch.equal(lb.zeropower_via_newtonschulz5(view, steps), lb.zeropower_via_newtonschulz5(plain.detach(), steps))
        got, want = (torch.autograd.grad(lb.zeropower_via_newtonschulz5(t, steps), t, d)[0] for t in (leaf, plain))
        assert torch.equal(got, want)
    lb.synchronize_and_check()


def test_c_abi_takes_four_elements_and_refuses_less():
    """bf16 gradients on 8 bytes go to the kernels that read 8 bytes at a time: the same values."""
    import ctypes as C
    import lact_b200 as lb
    from lact_b200 import _lib as L
    B, R, Cc = 2, 64, 128
    buf = torch.randn(B * R * Cc + 8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(torch.bfloat16)
    need = C.c_size_t(0)
    L.check(L.lib().lact_newton_schulz_workspace_bytes(B, R, Cc, C.byref(need)), "bytes")
    ws = L.workspace(need.value, buf.device)
    x = torch.empty(B, R, Cc, dtype=torch.bfloat16, device="cuda")
    run = lambda s: L.lib().lact_newton_schulz(buf[s:].data_ptr(), L.LACT_BF16, x.data_ptr(), B, R, Cc, 5, 0, ws.data_ptr(), ws.numel(),
                                               L.stream_ptr())
    assert run(4) == 0
    want = lb.zeropower_via_newtonschulz5(buf[4:4 + B * R * Cc].clone().view(B, R, Cc))
    assert torch.equal(x, want)
    with pytest.raises(ValueError):
        L.check(run(1), "lact_newton_schulz")
