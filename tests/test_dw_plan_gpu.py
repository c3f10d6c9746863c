"""GPU: weight gradients whose plan keeps whole blocks for the full waves and splits the rest (written partly by the CTAs, partly by
the reduction), in one call and as the weights part alone, against the oracle evaluated on the GPU in fp64."""
import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Hk,S,dh,E,de", [(1, 16, 16, 2560, 64, 11, 128), (2, 8, 8, 2500, 128, 11, 128), (1, 16, 16, 2560, 96, 7, 192)])
@pytest.mark.parametrize("parts", ["all", "weights"])
def test_whole_blocks_and_split_rest(B, H, Hk, S, dh, E, de, parts):
    import flashmhf_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(S)
    Q, dO = (torch.randn(B, H, S, dh, device="cuda", generator=g).bfloat16() for _ in range(2))
    K, U, V = (torch.randn(Hk, E, de, dh, device="cuda", generator=g).mul(0.1).bfloat16() for _ in range(3))
    R = torch.rand(B, H, S, E, device="cuda", generator=g)
    out = [torch.full_like(t, float("nan")) for t in (K, U, V)]
    fm.backward_raw(Q, K, U, V, R, dO, parts=parts, weight_grads=out)
    ref = orc.mhffn_backward(*(t.double() for t in (Q, K, U, V, R, dO)))[1:4]
    for name, a, b in zip("dK dU dV".split(), out, ref):
        assert orc.rel_l2(a.double(), b) < 1e-2, name
    fm.check_device_status()
