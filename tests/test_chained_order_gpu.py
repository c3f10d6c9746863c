"""GPU: a chained call reads its weights before the call ahead of it has ended.  What it may rely on is that the operation DIRECTLY before
it does not write them; weights written one operation earlier, in front of a plain, a chained or a split call, have to be seen."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("between", ["plain", "chained"])
@pytest.mark.parametrize("S", [8, 3000])     # with and without the split reduction behind the forward
def test_weights_written_two_operations_before(between, S):
    import flashmhf_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(S)
    rnd = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=g).mul_(std).bfloat16()
    H, E, de, dh = 8, 11, 256, 128
    Q, R = rnd(1, H, S, dh), torch.rand(1, H, S, E, device="cuda", generator=g)
    other = [rnd(H, E, de, dh, std=0.05) for _ in range(3)]
    sets = [[rnd(H, E, de, dh, std=0.05) for _ in range(3)] for _ in range(3)]
    want = [fm.forward_raw(Q, *w, R) for w in sets]
    torch.cuda.synchronize()
    live = [torch.empty_like(t) for t in sets[0]]
    for i in range(30):
        for dst, src in zip(live, sets[i % 3]):
            dst.copy_(src)
        fm.forward_raw(Q, *other, R, chained=between == "chained")
        assert torch.equal(fm.forward_raw(Q, *live, R, chained=True), want[i % 3])
    fm.check_device_status()
