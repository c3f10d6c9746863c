"""GPU: the head scaling in every form of the forward (split over the sub-networks, single token tiles, pairs of tiles), in dQ and in dR, element
by element against the oracle in fp64; and at the ends of the ranges of what it meets: subnormal Q, a large up scaling over small routing weights."""
import ctypes as C

import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


def _check(ins, scaling):
    import flashmhf_b200 as fm
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


# B, H, H_kuv, S, E, d_e and whether the forward splits the sub-networks.  On 148 SMs: 16 tiles, split; 100 tiles of 100 heads, single (in pairs
# they would take two rounds); 160 tiles of 8 heads, in pairs at d_h = 96 and 128
SHAPES = [((2, 4, 2, 200, 3, 128), True), ((1, 100, 50, 90, 1, 64), False), ((2, 8, 4, 1200, 2, 64), False)]


def _inputs(shape, dh, **kw):
    B, H, Hk, S, E, de = shape
    return [t.cuda() for t in orc.make_op_inputs(B, H, S, dh, E, de, Hkuv=Hk, seed=dh, dtype=torch.bfloat16, **kw)]


@pytest.mark.parametrize("dh", [64, 96, 128])
@pytest.mark.parametrize("head", [0.25, 0.5, 1.0, 2.0, 4.0, 1.7])
@pytest.mark.parametrize("shape,split", SHAPES)
def test_forward_and_input_gradients(lib, dh, head, shape, split):
    from flashmhf_b200 import _lib
    B, H, Hk, S, E, de = shape
    assert (lib.flashmhf_forward_workspace_bytes(C.byref(_lib.Dims(B, H, S, dh, Hk, E, de, 0))) > 0) == split
    _check(_inputs(shape, dh), (head, 0.6, 0.8))


@pytest.mark.parametrize("dh", [64, 96, 128])
@pytest.mark.parametrize("shape", [s for s, _ in SHAPES])
def test_subnormal_q(dh, shape):
    # odd multiples of the smallest bf16: half of one is not a bf16.  K, U and R bring the products back into the middle of fp32.
    Q, K, U, V, R, dO = _inputs(shape, dh, w_std=1.0)
    g = torch.Generator(device="cuda").manual_seed(1)
    bits = 2 * torch.randint(0, 8, Q.shape, device="cuda", generator=g) + 1
    Q = torch.where(Q > 0, bits, bits - 32768).to(torch.int16).view(torch.bfloat16)
    for head in (0.5, 1.0, 2.0, 1.7):
        _check([Q, K * 2.0 ** 60, U * 2.0 ** 80, V, R * 2.0 ** 60, dO], (head, 0.6, 0.8))


@pytest.mark.parametrize("dh", [64, 96, 128])
@pytest.mark.parametrize("shape", [s for s, _ in SHAPES])
def test_large_scaling_over_small_weights(dh, shape):
    # the constants' product is 2^125: any factor above 4 on it would overflow
    Q, K, U, V, R, dO = _inputs(shape, dh)
    _check([Q, K, U, V, R * 2.0 ** -120, dO * 2.0 ** -20], (0.5, 2.0 ** 126, 1.0))
