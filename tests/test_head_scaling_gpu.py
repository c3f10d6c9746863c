"""GPU: head scalings whose half is 1/4, 1/2 or 1 are applied to Q on its way to tensor memory, others to the products: forward, dQ and dR on both
sides of that rule and at its ends, element by element against the oracle in fp64."""
import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh", [64, 96, 128])
@pytest.mark.parametrize("head", [0.25, 0.5, 1.0, 2.0, 4.0, 1.7])
def test_forward_and_input_gradients(dh, head):
    import flashmhf_b200 as fm
    ins = [t.cuda() for t in orc.make_op_inputs(2, 4, 200, dh, 3, 128, Hkuv=2, seed=dh, dtype=torch.bfloat16)]
    scaling = (head, 0.6, 0.8)
    names = dict(zip(("head_scaling", "up_scaling", "final_scaling"), scaling))
    d = [t.double() for t in ins]
    O = fm.forward_raw(*ins[:5], scaling=scaling)
    dQ, *_, dR = fm.backward_raw(*ins, scaling=scaling, parts="inputs")
    ref = orc.mhffn_backward(*d, **names)
    # bf16 operands and results: about 2^-9 of the rms each; a wrong power of two would be off by the rms itself.  dR is summed in fp32 from
    # fp32 products of tanh.approx (2^-11 of a value each)
    for name, a, b in (("O", O, orc.mhffn_forward(*d[:5], **names)), ("dQ", dQ, ref[0]), ("dR", dR, ref[4])):
        assert orc.rel_l2(a.double(), b) < 1e-2, name
        assert orc.worst_element(a, b) < 0.05, name
    fm.check_device_status()
