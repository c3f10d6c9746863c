"""GPU: a training step of the layer element by element, over all head dimensions, more than one wave of CTAs, ragged lengths and batches of 1
to 16: y and the expert weights' gradients against the operator's oracle in fp64 on the layer's own intermediates, the other gradients against
the layer put together from its parts, and every gradient bit for bit on later steps with another input in between."""
import pytest
import torch
import torch.nn.functional as F

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,H,Hkuv,E,de,dh", [(5, 1645, 8, 8, 6, 256, 128), (1, 333, 8, 4, 5, 192, 128), (16, 130, 16, 16, 4, 320, 128),
                                                (3, 1031, 8, 8, 8, 256, 96), (7, 200, 8, 4, 5, 64, 96), (4, 2050, 8, 8, 6, 192, 64)])
def test_training_step(B, S, H, Hkuv, E, de, dh):
    import flashmhf_b200 as fm
    hid, g = H * dh, torch.Generator(device="cuda").manual_seed(S + dh)
    rnd = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=g).mul_(std).bfloat16()
    p = {n: rnd(E * de, Hkuv * dh, std=0.02) for n in ("gate_weight", "up_weight", "down_weight")}
    p.update(router=rnd(H, dh, E, std=0.1), q_norm=1 + rnd(H, dh, std=0.1), w_self=rnd(hid, hid, std=0.03), w_self_2=rnd(hid, hid, std=0.03))
    for t in p.values():
        t.requires_grad_(True)
    xs = [rnd(B, S, hid).requires_grad_(True) for _ in range(2)]
    dy = rnd(B, S, hid)

    def step(x):
        y = fm.mhffn_layer(x, p, H=H, Hkuv=Hkuv, E=E, apply_rmsnorm=True)
        return (y.detach(),) + torch.autograd.grad(y, [x, *p.values()], dy)

    names = ["y", "x", *p]
    first = step(xs[0])
    for _ in range(5):
        step(xs[1])
        for name, a, b in zip(names, step(xs[0]), first):
            assert torch.equal(a, b), name

    Q, R = fm.fused_prologue(F.linear(xs[0], p["w_self"]), p["q_norm"], p["router"])
    views = fm.expert_views(p["gate_weight"], p["up_weight"], p["down_weight"], Hkuv, E)
    y = F.linear(fm.flash_mhf(Q, *views, R).transpose(1, 2).reshape(B, S, hid), p["w_self_2"])
    want = dict(zip(names, (y.detach(),) + torch.autograd.grad(y, [xs[0], *p.values()], dy)))
    with torch.no_grad():
        ins = [t.double() for t in (Q, *views, R)]
        dO = (dy.view(-1, hid) @ p["w_self_2"]).view(B, S, H, dh).transpose(1, 2).double()
        O = orc.mhffn_forward(*ins).transpose(1, 2).reshape(B, S, hid)
        want["y"] = F.linear(O, p["w_self_2"].double())
        for name, t in zip(("gate_weight", "up_weight", "down_weight"), orc.mhffn_backward(*ins, dO)[1:4]):
            want[name] = t.permute(1, 2, 0, 3).reshape(E * de, Hkuv * dh)
    for name, a in zip(names, first):
        assert orc.worst_element(a, want[name]) < 0.05, name
    fm.check_device_status()
