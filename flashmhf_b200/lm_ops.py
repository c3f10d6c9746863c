"""Autograd wrappers of the two LM helper kernels (rotary embedding, hidden-size RMSNorm) in csrc/lm_aux.cu.

They serve flashmhf_b200/lm.py on CUDA bf16 tensors; the module keeps plain torch expressions for
everything else.  Both follow the reference's arithmetic (models/flashmhf/modeling_mhffnmoe.py:82-87,
:178-206) in fp32 with one rounding to bf16."""
from . import _lib

NORM_SIZES = (768, 1024, 2048)


class RotaryFunction:
    """x [B,S,heads,head_dim] bf16 contiguous, cos/sin fp32 [S, head_dim/2] -> rotated tensor of the same layout."""

    @staticmethod
    def apply(x, cos_t, sin_t):
        return _lib.native().rotary(x, cos_t, sin_t)


class RMSNormFunction:
    """x [..., n] bf16, weight [n] (any float dtype) -> y; n in NORM_SIZES."""

    @staticmethod
    def apply(x, weight, eps):
        return _lib.native().rmsnorm(x, weight, eps)


def rotary_pair(q, k, cos_t, sin_t):
    """(q, k) [B,S,heads,head_dim] bf16, rotated in one launch."""
    return _lib.native().rotary_pair(q, k, cos_t, sin_t)


def attention(x, wq, wk, wv, wo, num_heads, num_kv_heads, cos_t, sin_t):
    """Causal self-attention of x [B,S,hidden] bf16 with rotary embedding, without gradients (lm.Attention.forward's steps)."""
    return _lib.native().lm_attention(x, wq, wk, wv, wo, num_heads, num_kv_heads, cos_t, sin_t)


def add_rmsnorm(h, d, weight, eps):
    """(h + d, RMSNorm(h + d) * weight) for bf16 [..., n], n in NORM_SIZES, in one pass."""
    return _lib.native().add_rmsnorm(h, d, weight, eps)


def rotary_tables_f32(cos, sin):
    """The first half of the reference's (duplicated) cos/sin tables, as the fp32 values of their bf16 roundings."""
    h = cos.shape[-1] // 2
    return cos[:, :h].float().contiguous(), sin[:, :h].float().contiguous()
