"""Calls from a thread on which no CUDA context is current yet (all memory from torch's cache), against the oracle."""
import threading

import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dh,de", [(64, 64), (128, 128)])
def test_first_call_of_a_thread(dh, de):
    from flashmhf_b200 import functional as F
    Q, K, U, V, R, dO = orc.make_op_inputs(1, 2, 200, dh, 2, de, seed=0, dtype=torch.bfloat16)
    ins = [t.cuda() for t in (Q, K, U, V, R)]
    g = dO.cuda()
    F.forward_raw(*ins)       # fills torch's cache, so that the thread's allocations reach no CUDA call
    F.backward_raw(*ins, g)
    torch.cuda.synchronize()
    out, err = [], []

    def run():
        try:
            out.extend([F.forward_raw(*ins), *F.backward_raw(*ins, g)])
        except Exception as e:   # noqa: BLE001 - handed to the main thread
            err.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    assert not err, err
    torch.cuda.synchronize()
    f = [x.float() for x in (Q, K, U, V)]
    refs = [orc.mhffn_forward(*f, R), *orc.mhffn_backward(*(x.double() for x in f), R.double(), dO.double())]
    for a, r in zip(out, refs):
        assert orc.rel_l2(a.cpu().float(), r) < 1e-2
