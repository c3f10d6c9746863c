"""GPU: the layer's native call under the parts of autograd that look inside it: recomputation."""
import pytest
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu
KW = dict(H=4, Hkuv=2, E=3, apply_rmsnorm=True)


def _inputs(grad=True):
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s, std=0.05: torch.randn(*s, device="cuda", generator=g).mul(std).bfloat16().requires_grad_(grad)
    p = {n: rnd(192, 128) for n in ("gate_weight", "up_weight", "down_weight")}
    p.update(router=rnd(4, 64, 3, std=0.3), q_norm=rnd(4, 64, std=1.0), w_self=rnd(256, 256), w_self_2=rnd(256, 256))
    return rnd(2, 75, 256, std=1.0), rnd(256, 256), p, rnd(2, 75, 256, std=1.0).detach()


def test_recomputed_in_backward():
    """Non-reentrant checkpointing recomputes the region when the first saved tensor is asked for, which is the layer's: the operations in
    front of it have to be recorded then."""
    import flashmhf_b200 as fm
    x, w0, p, dy = _inputs()
    leaves = [x, w0, *p.values()]
    fn = lambda t: fm.mhffn_layer(F.silu(F.linear(t, w0)), p, **KW)
    want = torch.autograd.grad(fn(x), leaves, dy)
    got = torch.autograd.grad(checkpoint(fn, x, use_reentrant=False), leaves, dy)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
