"""GPU: the forward at d_h = 96 and 128 in pairs of CTAs, which share one head's weights: an odd number of token tiles of a head (half a pair
is empty, and a pair takes the last tile of one sequence and the first of the next), one work item of a pair and several, one 64-row block
per item, shared K/U/V heads, Q as a strided view, the chained entry point -- element by element against the oracle in fp64, weights in DRAM
and in L2; and a shape where single tiles need fewer rounds."""
import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh", [96, 128])
@pytest.mark.parametrize("chained", [False, True])
@pytest.mark.parametrize("B,H,Hk,S,E,de", [(3, 16, 16, 600, 2, 64), (5, 8, 4, 1100, 1, 64), (9, 16, 8, 77, 3, 192), (1, 16, 16, 1024, 1, 64),
                                           (1, 16, 16, 1025, 2, 64)])
@pytest.mark.parametrize("scaling", [(1.0, 1.0, 1.0), (8 ** 0.5, 0.7, 0.6)])
def test_forward(dh, chained, B, H, Hk, S, E, de, scaling):
    import flashmhf_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(S + dh + E)
    rnd = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=g).mul_(std).bfloat16()
    Q = rnd(B, S, H, dh).transpose(1, 2)
    K, U, V = (rnd(Hk, E, de, dh, std=0.1) for _ in range(3))
    R = torch.rand(B, H, S, E, device="cuda", generator=g)
    evict = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    first = fm.forward_raw(Q, K, U, V, R, scaling=scaling, chained=chained)
    for i in range(6):
        if i % 2 == 0:
            evict.zero_()
        assert torch.equal(fm.forward_raw(Q, K, U, V, R, scaling=scaling, chained=chained), first)
    ref = orc.mhffn_forward(*(t.double() for t in (Q, K, U, V, R)), **dict(zip(("head_scaling", "up_scaling", "final_scaling"), scaling)))
    # bf16 operands and result (2^-9 of each term, about 2^-9 of the rms together); a tile of the wrong weights is off by the rms itself
    assert orc.worst_element(first, ref) < 0.05
    fm.check_device_status()
