"""GPU: weight gradients whose plan keeps whole blocks for the full waves and splits the rest (written partly by the CTAs, partly by
the reduction), or cuts some blocks unevenly, in one call and as the weights part alone, against the oracle evaluated on the GPU in fp64."""
import ctypes as C

import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


WHOLE = [(1, 16, 16, 2560, 64, 11, 128), (2, 8, 8, 2500, 128, 11, 128), (1, 16, 16, 2560, 96, 7, 192)]
UNEVEN = [(3, 16, 16, 1196, 64, 9, 64), (4, 4, 2, 387, 128, 19, 128), (7, 16, 16, 489, 96, 9, 64)]


@pytest.mark.parametrize("B,H,Hk,S,dh,E,de", WHOLE + UNEVEN)
@pytest.mark.parametrize("parts", ["all", "weights"])
def test_whole_blocks_and_split_rest(B, H, Hk, S, dh, E, de, parts):
    import flashmhf_b200 as fm
    from flashmhf_b200 import _lib
    plan = _lib.BackwardPlan()
    assert _lib.load().flashmhf_backward_plan(C.byref(_lib.Dims(B, H, S, dh, Hk, E, de, _lib.BF16)), 0 if parts == "all" else _lib.BWD_WEIGHTS,
                                              C.byref(plan)) == 0
    assert plan.splits > 1 and (plan.whole_blocks if (B, H, Hk, S, dh, E, de) in WHOLE else plan.uneven_blocks) > 0
    g = torch.Generator(device="cuda").manual_seed(S)
    Q, dO = (torch.randn(B, H, S, dh, device="cuda", generator=g).bfloat16() for _ in range(2))
    K, U, V = (torch.randn(Hk, E, de, dh, device="cuda", generator=g).mul(0.1).bfloat16() for _ in range(3))
    R = torch.rand(B, H, S, E, device="cuda", generator=g)
    out = [torch.full_like(t, float("nan")) for t in (K, U, V)]
    fm.backward_raw(Q, K, U, V, R, dO, parts=parts, weight_grads=out)
    ref = orc.mhffn_backward(*(t.double() for t in (Q, K, U, V, R, dO)))[1:4]
    for name, a, b in zip("dK dU dV".split(), out, ref):
        assert orc.rel_l2(a.double(), b) < 1e-2, name
        assert orc.worst_element(a, b) < 0.05, name
    fm.check_device_status()
