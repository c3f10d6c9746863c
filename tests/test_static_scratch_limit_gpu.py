"""GPU: flashmhf_backward_static_scratch where the plan of flashmhf_backward wants more partial sums than the built-in array holds: the call
runs with fewer parts.  Against flashmhf_backward, element by element: fp32 sums in another order, so a bf16 result one step (2^-8) away
at most, of values whose terms cancel a few steps of the rms."""
import ctypes as C

import pytest
import torch

from oracle import mhffn_oracle as orc
from tests.test_zz_no_alloc import _static_backward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,S,dh,Hk,E,de", [(7, 8, 1442, 64, 8, 20, 320), (6, 8, 2439, 96, 4, 20, 128), (7, 16, 671, 128, 8, 10, 320)])
def test_fewer_parts_where_the_sums_do_not_fit(B, H, S, dh, Hk, E, de):
    import flashmhf_b200 as fm
    from flashmhf_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(S)
    Q, dO = (torch.randn(B, H, S, dh, device="cuda", generator=g).bfloat16() for _ in range(2))
    K, U, V = (torch.randn(Hk, E, de, dh, device="cuda", generator=g).mul(0.05).bfloat16() for _ in range(3))
    R = torch.rand(B, H, S, E, device="cuda", generator=g)
    d = _lib.Dims(B, H, S, dh, Hk, E, de, _lib.BF16)
    assert _lib.load().flashmhf_backward_workspace_bytes(C.byref(d)) > _lib.STATIC_SCRATCH_BYTES >= 12 * Hk * E * de * dh
    want = fm.backward_raw(Q, K, U, V, R, dO)
    got, _ = _static_backward(Q, K, U, V, R, dO)
    for name, a, b in zip("dQ dK dU dV dR".split(), got, want):
        assert orc.worst_element(a, b) < 0.02, name
