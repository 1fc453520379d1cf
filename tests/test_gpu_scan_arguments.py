"""Arguments of the recurrence that reach past its usual form."""
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
