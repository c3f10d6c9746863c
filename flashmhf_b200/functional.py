"""The operator's Python entry points: torch tensors in, C-ABI calls out.

``flash_mhf(Q, K, U, V, R)`` has the call signature of the reference's
``FlashMLPFunction.apply`` (kernels/triton/flash_mlp_moe.py:739-868) and of its ThunderKittens
twin (kernels/thunderkittens/flash_ffn_moe_torch.py:5-24): it saves the five inputs, keeps no
intermediate, and recomputes in backward.  Checks, allocations and autograd run in the native host module
(csrc/torch_host.cpp), all arithmetic in the CUDA library; PyTorch supplies device memory and the current stream."""
import torch

from . import _lib

_DT = {torch.bfloat16: _lib.BF16, torch.float32: _lib.F32_CHECK}


def _tensor(t):
    s = t.stride()
    return _lib.Tensor(t.data_ptr(), (s[0], s[1], s[2]))


def _dims(B, H, S, dh, hk, E, de, dtype):
    return _lib.Dims(B, H, S, dh, hk, E, de, _DT[dtype])


def forward_raw(Q, K, U, V, R, out=None, scaling=_lib.NO_SCALING, chained=False, workspace=None):
    """O = flashmhf_forward(...) on the current stream; no autograd.

    ``chained``: use ``flashmhf_forward_chained`` -- for back-to-back calls over constant weights (a decode loop,
    usually replayed from a CUDA graph): the call may start, and stream in its first weight tiles, while the kernel
    before it on the stream still runs.  The caller promises that K, U, V are not written by the operation directly
    before the call.  Same result, bit for bit.
    ``workspace``: optional uint8 tensor to use as the call's scratch (at least ``flashmhf_forward_workspace_bytes``)."""
    hs, us, fs = scaling
    return _lib.native().op_forward(Q, K, U, V, R, out, hs, us, fs, chained, workspace)


_PARTS = {"all": 0, "inputs": _lib.BWD_INPUTS, "weights": _lib.BWD_WEIGHTS}


def backward_raw(Q, K, U, V, R, dO, scaling=_lib.NO_SCALING, parts="all", weight_grads=None):
    """(dQ, dK, dU, dV, dR) = flashmhf_backward(...) on the current stream; no autograd.

    ``parts``: "all", or "weights" (dK, dU, dV only; dQ and dR come back as None) or "inputs" (the reverse) --
    data-parallel training runs the weights part first and overlaps its all-reduce with the inputs part.
    ``weight_grads``: optional (dK, dU, dV) tensors to write into (e.g. three views of one all-reduce bucket)."""
    if dO.shape != Q.shape:
        raise AssertionError("grad_output shape should be the same as Q")
    if parts not in _PARTS:
        raise ValueError(f"parts must be 'all', 'weights' or 'inputs', got {parts!r}")
    hs, us, fs = scaling
    return _lib.native().op_backward(Q, K, U, V, R, dO, hs, us, fs, _PARTS[parts], None if weight_grads is None else list(weight_grads))


class FlashMHFFunction(torch.autograd.Function):
    """apply(Q, K, U, V, R[, head_scaling, up_scaling, final_scaling]) -> O, differentiable in the five tensors.

    The constants are those of the reference's eager loop (models/flashmhf/modeling_mhffnmoe.py:270-279, 420-425);
    its own flash path has none (kernels/triton/flash_mlp_moe.py:741), which is the default of 1.
    ``apply`` goes to the native autograd function; ``forward`` / ``backward`` are the same two calls for a caller that
    builds its own autograd function from them."""

    @staticmethod
    def forward(ctx, Q, K, U, V, R, head_scaling=1.0, up_scaling=1.0, final_scaling=1.0):
        ctx.scaling = (float(head_scaling), float(up_scaling), float(final_scaling))
        O = forward_raw(Q, K, U, V, R, scaling=ctx.scaling)
        ctx.save_for_backward(Q, K, U, V, R)
        return O

    @staticmethod
    def backward(ctx, grad_output):
        Q, K, U, V, R = ctx.saved_tensors
        dQ, dK, dU, dV, dR = backward_raw(Q, K, U, V, R, grad_output, scaling=ctx.scaling)
        return dQ, dK, dU, dV, dR.to(R.dtype), None, None, None

    @staticmethod
    def apply(Q, K, U, V, R, head_scaling=1.0, up_scaling=1.0, final_scaling=1.0):
        return _lib.native().flash_mhf(Q, K, U, V, R, head_scaling, up_scaling, final_scaling)


def flash_mhf(Q, K, U, V, R, head_scaling=1.0, up_scaling=1.0, final_scaling=1.0):
    return _lib.native().flash_mhf(Q, K, U, V, R, head_scaling, up_scaling, final_scaling)


def check_device_status():
    """Synchronise and raise FlashMHFError if a kernel of this library gave up on a bounded wait (its outputs are then
    unwritten).  The entry points only enqueue work, so this is the place a host loop learns of it: call it where the
    loop synchronises anyway (after the loss is read back, at the end of a step)."""
    _lib.device_status()
