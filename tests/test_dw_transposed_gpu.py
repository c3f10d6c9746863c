"""GPU: the weight-gradient kernel of d_h = 64 and 96 where it can go wrong: an odd number of 64-row weight blocks (its CTAs own
128 rows), sub-networks of 64 rows (128 rows touch two of them), token counts around its 64-token tiles, shared K/U/V heads, one
tile and many splits -- against the oracle in fp64, and bit for bit on a second call into poisoned outputs."""
import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh", [64, 96])
@pytest.mark.parametrize("B,H,Hk,S,E,de", [(1, 1, 1, 1, 1, 64), (1, 2, 2, 63, 3, 64), (2, 2, 1, 64, 2, 64), (1, 2, 2, 65, 5, 64),
                                           (3, 4, 2, 130, 1, 192), (1, 1, 1, 3000, 1, 128), (2, 2, 2, 257, 7, 320)])
def test_weight_gradients(dh, B, H, Hk, S, E, de):
    import flashmhf_b200 as fm
    ins = [t.cuda() for t in orc.make_op_inputs(B, H, S, dh, E, de, Hkuv=Hk, seed=S + E, dtype=torch.bfloat16)]
    got = fm.backward_raw(*ins, parts="weights")[1:4]
    ref = orc.mhffn_backward(*(t.cpu().double() for t in ins))[1:4]
    for name, a, b in zip("dK dU dV".split(), got, ref):
        assert orc.rel_l2(a.cpu().double(), b) < 1e-2, name
        assert orc.worst_element(a.cpu(), b) < 0.05, name
    again = [torch.full_like(t, float("nan")) for t in ins[1:4]]
    fm.backward_raw(*ins, parts="weights", weight_grads=again)
    for a, b in zip(got, again):
        assert torch.equal(a, b)
    fm.check_device_status()
