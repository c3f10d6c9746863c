"""GPU: the layer as one autograd node (bf16 everywhere) against the same layer put together from its parts, whose parity
with the oracle other tests check: with and without RMSNorm, biases and projections, parameters read as bf16 or fp32, and
gradients asked for in part only."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("norm,proj,bias,fp32_router,frozen", [
    (True, True, False, False, ()), (False, True, True, False, ()), (True, False, False, False, ()), (True, True, False, True, ()),
    (True, True, True, False, ("gate_weight", "up_weight", "down_weight")),
    (False, True, False, False, ("x", "w_self", "router")), (True, True, False, False, ("w_self_2", "router", "q_norm"))])
def test_layer_node_equals_its_parts(norm, proj, bias, fp32_router, frozen):
    import flashmhf_b200 as fm
    B, S, H, Hkuv, E, de, dh = 2, 75, 4, 2, 3, 64, 64
    hid, g = H * dh, torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s, std=0.05: torch.randn(*s, device="cuda", generator=g).mul(std).bfloat16()
    p = {"gate_weight": rnd(E * de, Hkuv * dh), "up_weight": rnd(E * de, Hkuv * dh), "down_weight": rnd(E * de, Hkuv * dh),
         "router": rnd(H, dh, E, std=0.3), "q_norm": 1 + rnd(H, dh)}
    if fp32_router:
        p["router"] = p["router"].float()
    if proj:
        p.update(w_self=rnd(hid, hid), w_self_2=rnd(hid, hid))
    if bias:
        p.update(w_self_bias=rnd(hid), w_self_2_bias=rnd(hid))
    if not norm:
        del p["q_norm"]
    x, dy = rnd(B, S, hid, std=1.0), rnd(B, S, hid, std=1.0)
    leaves = {"x": x, **p}
    leaves = {k: v.requires_grad_(True) for k, v in leaves.items() if k not in frozen}
    y = fm.mhffn_layer(x, p, H=H, Hkuv=Hkuv, E=E, apply_rmsnorm=norm)
    got = torch.autograd.grad(y, list(leaves.values()), dy)
    q = F.linear(x, p["w_self"], p.get("w_self_bias")) if proj else x
    Q, R = fm.fused_prologue(q, p.get("q_norm"), p["router"].float())
    O = fm.flash_mhf(Q, *fm.expert_views(p["gate_weight"], p["up_weight"], p["down_weight"], Hkuv, E), R)
    O = O.transpose(1, 2).reshape(B, S, hid)
    want_y = F.linear(O, p["w_self_2"], p.get("w_self_2_bias")) if proj else O
    want = torch.autograd.grad(want_y, list(leaves.values()), dy)
    assert _rel(y, want_y) < 1e-3
    for name, a, b in zip(leaves, got, want):
        assert a.dtype == b.dtype and a.shape == b.shape, name
        assert _rel(a, b) < 5e-3, name
    fm.check_device_status()


def test_parameters_that_do_not_fit_are_refused():
    """Before their addresses go to a kernel."""
    import flashmhf_b200 as fm
    x = torch.zeros(1, 4, 256, device="cuda", dtype=torch.bfloat16)
    router, norm = torch.zeros(4, 64, 2, device="cuda"), torch.ones(4, 64, device="cuda")
    for r, n in ((router.cpu(), norm), (router, norm.cpu()), (router, norm[:2])):
        with pytest.raises(ValueError):
            fm.fused_prologue(x, n, r)
