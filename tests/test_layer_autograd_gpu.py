"""GPU: the layer's native call under the parts of autograd that look inside it: recomputation, saved-tensor hooks and forward mode."""
import pytest
import torch
import torch.nn.functional as F
import torch.autograd.forward_ad as fwAD
from torch.utils.checkpoint import checkpoint

from oracle import mhffn_oracle as orc

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


def test_saved_tensors_come_back_in_another_layout():
    """What an unpack hook returns has the values and the shape of what was saved; its strides may be others."""
    import flashmhf_b200 as fm
    x, _, p, dy = _inputs()
    leaves = [x, *p.values()]
    want = torch.autograd.grad(fm.mhffn_layer(x, p, **KW), leaves, dy)
    turn = lambda t: t.transpose(-1, -2).contiguous().transpose(-1, -2) if t.dim() > 1 else t
    with torch.autograd.graph.saved_tensors_hooks(turn, lambda t: t):
        y = fm.mhffn_layer(x, p, **KW)
    got = torch.autograd.grad(y, leaves, dy)
    for a, b in zip(got, want):
        assert orc.rel_l2(a, b) < 1e-3   # (a library product may round otherwise for another layout)


@pytest.mark.parametrize("grad", [False, True])
def test_forward_mode_is_refused(grad):
    """There is no forward-mode derivative: an input that carries a tangent is an error, not a result without one."""
    import flashmhf_b200 as fm
    from flashmhf_b200 import lm, lm_ops
    x, _, p, _ = _inputs(False)
    with torch.set_grad_enabled(grad), fwAD.dual_level():
        for name in ("x", "router", "gate_weight"):
            q = dict(p)
            t = x if name == "x" else p[name]
            dual = fwAD.make_dual(t, torch.ones_like(t))
            if name != "x":
                q[name] = dual
            with pytest.raises((RuntimeError, NotImplementedError)):
                fm.mhffn_layer(dual if name == "x" else x, q, **KW)
    cfg = lm.LMConfig(hidden_size=256, num_attention_heads=4, num_key_value_heads=4)
    att = lm.Attention(cfg).cuda().bfloat16()
    cos, sin = lm.rotary_tables(75, 64, 10000.0, x.device, torch.bfloat16)
    with torch.set_grad_enabled(grad), fwAD.dual_level():
        with pytest.raises((RuntimeError, NotImplementedError)):
            att(fwAD.make_dual(x, torch.ones_like(x)), cos, sin, tables=lm_ops.rotary_tables_f32(cos, sin))
