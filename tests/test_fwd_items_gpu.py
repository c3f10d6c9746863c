"""GPU: the forward where a CTA walks several work items (token tiles): each item's Q replaces the last one's in tensor memory, which must
wait for every product of the item before, those of the other activation team included.  Even and odd numbers of 64-row blocks per
item, one block among them, ragged last tiles; element by element against the oracle in fp64, weights in DRAM and in L2."""
import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh", [64, 96, 128])
@pytest.mark.parametrize("B,H,Hk,S,E,de", [(4, 16, 16, 1000, 1, 64), (3, 16, 8, 1153, 2, 64), (4, 16, 16, 1000, 3, 64), (3, 16, 16, 1153, 5, 192),
                                           (2, 16, 16, 2300, 4, 256)])
def test_forward_over_several_items_per_cta(dh, B, H, Hk, S, E, de):
    import flashmhf_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(S + dh + E)
    rnd = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=g).mul_(std).bfloat16()
    Q = rnd(B, H, S, dh)
    K, U, V = (rnd(Hk, E, de, dh, std=0.1) for _ in range(3))
    R = torch.rand(B, H, S, E, device="cuda", generator=g)
    evict = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    first = fm.forward_raw(Q, K, U, V, R)
    for i in range(8):
        if i % 2 == 0:
            evict.zero_()
        assert torch.equal(fm.forward_raw(Q, K, U, V, R), first)
    ref = orc.mhffn_forward(*(t.double() for t in (Q, K, U, V, R)))
    # bf16 operands and result (2^-9 of each term, about 2^-9 of the rms together); a tile of the wrong Q is off by the rms itself
    assert orc.worst_element(first, ref) < 0.05
    fm.check_device_status()
