"""The FFN layer around the operator, with the fused prologue.

``fused_prologue`` replaces what the reference layer does between its first projection and the
operator (models/flashmhf/modeling_mhffnmoe.py:362-386): head split, per-head RMSNorm, the
transposing copy of Q, and the router weights.  One CUDA kernel reads the projected activations
in their own [B,S,H,d_h] layout and writes the normalised Q in the same layout plus R; the operator
then reads Q in place through strides and writes O in that layout too, so the two
``transpose(1,2).contiguous()`` copies of the reference (modeling:374, 408) vanish.

``mhffn_layer`` is the whole layer (modeling:352-431) built from it; parameter names and shapes are the
reference's (w_self, w_self_2 [hid,hid]; gate/up/down_weight [I, H_kuv*d_h]; router [H,d_h,E];
q_norm [H,d_h]) so its state dicts load."""
import torch
import torch.nn.functional as F

from . import _lib
from .functional import flash_mhf


def fused_prologue(x_proj, q_norm, router, eps=1e-5):
    """(x_proj [B,S,H*d_h] bf16, q_norm [H,d_h] or None, router [H,d_h,E]) -> (Q [B,H,S,d_h] view, R [B,H,S,E] fp32)."""
    return _lib.native().fused_prologue(x_proj, q_norm, router, eps)


def torch_prologue(x_proj, q_norm, router, eps=1e-5):
    """The same two results from library element-wise kernels, for router shapes the fused kernels do not take (more
    than 32 sub-networks per head): per-head RMSNorm in fp32, Q as a [B,H,S,d_h] view, R = normalised sigmoid."""
    H, dh, _ = router.shape
    B, S, _ = x_proj.shape
    q = x_proj.view(B, S, H, dh)
    if q_norm is not None:
        qf = q.float()
        q = (qf * torch.rsqrt(qf.pow(2).mean(-1, keepdim=True) + eps) * q_norm.float()[None, None]).to(x_proj.dtype)
    Q = q.transpose(1, 2)
    R = (Q.float() @ router.float()).sigmoid()
    return Q, R / R.sum(dim=-1, keepdim=True).clamp(min=1e-20)


def expert_views(gate_weight, up_weight, down_weight, Hkuv, E):
    """[I, H_kuv*d_h] parameters -> [H_kuv, E, d_e, d_h] strided views the operator reads in place (no copy)."""
    I = gate_weight.shape[0]
    dh = gate_weight.shape[1] // Hkuv
    f = lambda w: w.view(E, I // E, Hkuv, dh).permute(2, 0, 1, 3)
    return f(gate_weight), f(up_weight), f(down_weight)


def mhffn_layer(x, p, *, H, Hkuv, E, apply_rmsnorm, eps=1e-5, head_scaling=1.0, up_scaling=1.0, final_scaling=1.0):
    """y = w_self_2(op(prologue(w_self(x)))) for bf16 CUDA tensors; p holds the reference's parameter names
    (optionally ``w_self_bias`` / ``w_self_2_bias``, the biases the reference creates with config.mlp_bias).
    The three constants are the eager layer's (models/flashmhf/modeling_mhffnmoe.py:270-279); every shipped
    configuration leaves them at 1."""
    w1, w2 = p.get("w_self"), p.get("w_self_2")
    b1 = p.get("w_self_bias") if w1 is not None else None
    b2 = p.get("w_self_2_bias") if w2 is not None else None
    q_norm = p["q_norm"] if apply_rmsnorm else None
    if p["router"].shape[-1] != E:
        raise ValueError(f"router must be [H, d_h, {E}], got {tuple(p['router'].shape)}")
    if E <= 32:
        return _lib.native().mhffn_layer(x, w1, b1, q_norm, p["router"], p["gate_weight"], p["up_weight"], p["down_weight"], w2, b2,
                                         Hkuv, eps, head_scaling, up_scaling, final_scaling)
    B, S, hid = x.shape
    q_lin = F.linear(x, w1, b1) if w1 is not None else x
    Q, R = torch_prologue(q_lin, q_norm, p["router"], eps)
    K, U, V = expert_views(p["gate_weight"], p["up_weight"], p["down_weight"], Hkuv, E)
    O = flash_mhf(Q, K, U, V, R, head_scaling, up_scaling, final_scaling)  # [B,H,S,d_h] view of [B,S,H,d_h] memory
    O = O.transpose(1, 2).reshape(B, S, hid)          # no copy when O kept Q's layout
    return F.linear(O, w2, b2) if w2 is not None else O
