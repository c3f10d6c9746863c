"""GPU: the weight-gradient kernel of d_h = 128 where it can go wrong: token counts around its 128-token tiles, one tile and many, one
64-row block and several sub-networks, shared K/U/V heads, the eager layer's constants, weights and tokens in DRAM and in L2 -- element by
element against the oracle in fp64, and bit for bit on later calls into poisoned outputs."""
import time

import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Hk,S,E,de", [(1, 1, 1, 1, 1, 64), (1, 2, 2, 127, 3, 64), (2, 2, 1, 128, 2, 64), (1, 2, 2, 129, 5, 64),
                                           (3, 4, 2, 257, 1, 192), (1, 1, 1, 3000, 1, 128), (5, 4, 4, 900, 7, 320)])
def test_weight_gradients(B, H, Hk, S, E, de):
    import flashmhf_b200 as fm
    ins = [t.cuda() for t in orc.make_op_inputs(B, H, S, 128, E, de, Hkuv=Hk, seed=S + E, dtype=torch.bfloat16)]
    scaling = (1.7, 0.6, 0.8)
    got = fm.backward_raw(*ins, scaling=scaling, parts="weights")[1:4]
    names = dict(zip(("head_scaling", "up_scaling", "final_scaling"), scaling))
    ref = orc.mhffn_backward(*(t.double() for t in ins), **names)[1:4]
    for name, a, b in zip("dK dU dV".split(), got, ref):
        # bf16 operands and results: 2^-9 of each term, together about 2^-9 of the rms; one wrong row or tile is off by the rms itself
        assert orc.rel_l2(a.double(), b) < 1e-2, name
        assert orc.worst_element(a, b) < 0.05, name
    evict = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    for i in range(6):
        if i % 2 == 0:
            evict.zero_()
        again = [torch.full_like(t, float("nan")) for t in ins[1:4]]
        fm.backward_raw(*ins, scaling=scaling, parts="weights", weight_grads=again)
        assert all(torch.equal(a, b) for a, b in zip(got, again))
    fm.check_device_status()


def test_tensor_maps_of_a_dozen_layers():
    # A thread keeps 64 encoded maps.  A weight-gradient call needs five (Q, dO, K, U, V), so twelve layers' fit; with maps of its own for K and U
    # it would need seven, and every call would encode all of them anew (8.7 us of host time a call instead of 7.3).
    import flashmhf_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    layers = [([rnd(1, 2, 128, 128)] + [rnd(2, 1, 64, 128) for _ in range(3)] + [torch.rand(1, 2, 128, 1, device="cuda")], rnd(1, 2, 128, 128),
               [rnd(2, 1, 64, 128) for _ in range(3)]) for _ in range(12)]

    def host_us(n):
        best = float("inf")
        for i in range(60):
            torch.cuda.synchronize()
            t = time.perf_counter()
            for ins, dO, grads in layers[:n]:
                fm.backward_raw(*ins, dO, parts="weights", weight_grads=grads)
            if i >= 10:
                best = min(best, (time.perf_counter() - t) / n)
        return best

    assert min(host_us(12) / host_us(6) for _ in range(5)) < 1.08   # 1.01 measured, 1.14 with seven maps; the host may be busy: the best of five
