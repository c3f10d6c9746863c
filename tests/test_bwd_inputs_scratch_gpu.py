"""GPU: scratch of a call for dQ and dR alone.  flashmhf_backward leaves workspace and workspace_bytes alone then (a caller may leave
them unset, or have another stream's call use that memory); flashmhf_backward_inputs splits short inputs with it."""
import ctypes as C

import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh", [64, 96, 128])
def test_inputs_alone(dh):
    import flashmhf_b200 as fm
    from flashmhf_b200 import _lib
    from flashmhf_b200.functional import _dims, _tensor
    lib = _lib.load()
    B, H, Hk, S, E, de = 2, 4, 2, 150, 5, 192
    Q, K, U, V, R, dO = (t.cuda() for t in orc.make_op_inputs(B, H, S, dh, E, de, Hkuv=Hk, seed=dh, dtype=torch.bfloat16))
    d = _dims(B, H, S, dh, Hk, E, de, Q.dtype)
    plan = _lib.BackwardPlan()
    assert lib.flashmhf_backward_plan(C.byref(d), _lib.BWD_INPUTS, C.byref(plan)) == 0 and plan.dq_splits > 1
    need = lib.flashmhf_backward_inputs_workspace_bytes(C.byref(d))
    assert need == plan.dq_splits * B * H * S * dh * 4
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    none = _lib.Tensor(None, (0, 0, 0))

    def call(fn, ptr, nbytes):
        dQ, dR = torch.full_like(Q, float("nan")), torch.full_like(R, float("nan"))
        p = _lib.BwdParams(d, *(_tensor(t) for t in (Q, K, U, V, R, dO)), _tensor(dQ), none, none, none, _tensor(dR), ptr, nbytes,
                           _lib.Scaling(1.0, 1.0, 1.0), _lib.BWD_INPUTS)
        rc = fn(C.byref(p), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        return rc, dQ, dR

    ws.fill_(0x5a)
    rc, dQ, dR = call(lib.flashmhf_backward, ws.data_ptr(), need)
    assert rc == 0 and bool((ws == 0x5a).all())
    for ptr, nbytes in ((None, 0), (ws.data_ptr(), need - 256)):
        rc, dQ1, dR1 = call(lib.flashmhf_backward_inputs, ptr, nbytes)
        assert rc == 0 and torch.equal(dQ, dQ1) and torch.equal(dR, dR1) and bool((ws == 0x5a).all())
    assert call(lib.flashmhf_backward_inputs, ws.data_ptr() + 16, need - 16)[0] == -6
    rc, dQ2, dR2 = call(lib.flashmhf_backward_inputs, ws.data_ptr(), need)
    assert rc == 0 and torch.equal(dR, dR2) and not bool((ws == 0x5a).all())
    want = orc.mhffn_backward(*(t.double() for t in (Q, K, U, V, R, dO)))
    assert orc.rel_l2(dQ, want[0]) < 1e-2 and orc.rel_l2(dQ2, want[0]) < 1e-2
    a, b = fm.backward_raw(Q, K, U, V, R, dO, parts="inputs"), fm.backward_raw(Q, K, U, V, R, dO)
    assert torch.equal(a[0], dQ2) and torch.equal(a[0], b[0]) and torch.equal(a[4], b[4])
