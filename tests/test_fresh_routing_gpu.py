"""GPU: the layer without gradients, whose operator starts under the prologue that still writes Q and R into reused memory: calls on new
activations, back to back, must give what each gives alone, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("B,S,H,Hkuv,E,de,dh", [(64, 1, 16, 16, 22, 256, 128), (3, 333, 8, 4, 5, 192, 128), (4, 700, 8, 8, 8, 256, 96),
                                                (2, 1100, 16, 16, 16, 192, 64)])
def test_back_to_back_layer_calls(grad, B, S, H, Hkuv, E, de, dh):
    import flashmhf_b200 as fm
    g, hid = torch.Generator(device="cuda").manual_seed(S + dh), H * dh
    rnd = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=g).mul_(std).bfloat16()
    p = {n: rnd(E * de, Hkuv * dh, std=0.05) for n in ("gate_weight", "up_weight", "down_weight")}
    p.update(router=rnd(H, dh, E, std=0.3), q_norm=1 + rnd(H, dh, std=0.1), w_self=rnd(hid, hid, std=0.03), w_self_2=rnd(hid, hid, std=0.03))
    if grad:
        p["router"].requires_grad_(True)
    xs = [rnd(B, S, hid, std=2.0 + i) for i in range(6)]
    call = lambda x: fm.mhffn_layer(x, p, H=H, Hkuv=Hkuv, E=E, apply_rmsnorm=True).detach()
    alone = []
    for x in xs:
        alone.append(call(x).clone())
        torch.cuda.synchronize()
    for _ in range(20):
        for want, got in zip(alone, [call(x) for x in xs]):
            assert torch.equal(want, got)
    fm.check_device_status()
