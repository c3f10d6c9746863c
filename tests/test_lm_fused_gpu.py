"""GPU: the two-in-one LM helpers against the single ones: rotary embedding of queries and keys in one launch, and the residual
addition joined with the RMSNorm behind it, forward and backward."""
import pytest
import torch

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,nq,nk,hd", [(2, 37, 4, 4, 64), (1, 130, 6, 2, 32)])
def test_rotary_pair_equals_two_single_calls(B, S, nq, nk, hd):
    from flashmhf_b200 import lm, lm_ops
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, gq, gk = (torch.randn(B, S, n, hd, device="cuda", generator=g).bfloat16() for n in (nq, nk, nq, nk))
    ct, st = lm_ops.rotary_tables_f32(*lm.rotary_tables(S, hd, 10000.0, q.device, torch.bfloat16))
    a, b = (t.clone().requires_grad_(True) for t in (q, k)), (t.clone().requires_grad_(True) for t in (q, k))
    a, b = tuple(a), tuple(b)
    pair = lm_ops.rotary_pair(*a, ct, st)
    single = tuple(lm_ops.RotaryFunction.apply(t, ct, st) for t in b)
    torch.autograd.backward(pair, (gq, gk))
    torch.autograd.backward(single, (gq, gk))
    for x, y in zip(pair + tuple(t.grad for t in a), single + tuple(t.grad for t in b)):
        assert torch.equal(x, y)
    only_k = k.clone().requires_grad_(True)
    lm_ops.rotary_pair(q, only_k, ct, st)[1].backward(gk)
    assert torch.equal(only_k.grad, b[1].grad)


@pytest.mark.parametrize("rows,n,wdt", [(5, 768, torch.bfloat16), (333, 1024, torch.float32), (77, 2048, torch.bfloat16)])
@pytest.mark.parametrize("use_sum", [True, False])
def test_add_rmsnorm_equals_addition_then_norm(rows, n, wdt, use_sum):
    from flashmhf_b200 import lm_ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, d, gy, gs = (torch.randn(rows, n, device="cuda", generator=g).bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(n, device="cuda", generator=g)).to(wdt)
    a, b = ([t.clone().requires_grad_(True) for t in (x, d, w)] for _ in range(2))
    s1, y1 = lm_ops.add_rmsnorm(*a, 1e-5)
    s2 = b[0] + b[1]
    y2 = lm_ops.RMSNormFunction.apply(s2, b[2], 1e-5)
    assert torch.equal(s1, s2) and torch.equal(y1, y2)
    if use_sum:
        torch.autograd.backward((s1, y1), (gs, gy))
        torch.autograd.backward((s2, y2), (gs, gy))
    else:
        y1.backward(gy)
        y2.backward(gy)
    for p, q in zip(a, b):
        assert orc.rel_l2(p.grad.float(), q.grad.float()) < 4e-3
    assert torch.equal(a[2].grad, b[2].grad)


@pytest.mark.parametrize("B,S,kv", [(1, 33, 4), (2, 130, 2)])
def test_attention_without_gradients_equals_the_module_path(B, S, kv):
    """lm.Attention takes one native call under no_grad and its own steps otherwise."""
    from flashmhf_b200 import lm, lm_ops
    torch.manual_seed(S)
    cfg = lm.LMConfig(hidden_size=256, num_attention_heads=4, num_key_value_heads=kv)
    att = lm.Attention(cfg).cuda().bfloat16()
    x = torch.randn(B, S, 256, device="cuda").bfloat16()
    cos, sin = lm.rotary_tables(S, 64, 10000.0, x.device, torch.bfloat16)
    tables = lm_ops.rotary_tables_f32(cos, sin)
    want = att(x, cos, sin, tables=tables).detach()
    with torch.no_grad():
        got = att(x, cos, sin, tables=tables)
    assert orc.rel_l2(got.float(), want.float()) < 1e-2


def test_sizes_that_do_not_fit_are_refused():
    """Before an address goes to a kernel; an addend that would have to be broadcast takes the separate steps."""
    from flashmhf_b200 import lm, lm_ops
    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    x, w = rnd(4, 6, 768), torch.ones(768, device="cuda", dtype=torch.bfloat16)
    for d in (rnd(1, 6, 768), rnd(4, 6, 767), rnd(4, 6, 768).float(), rnd(4, 6, 768).cpu()):
        with pytest.raises(ValueError):
            lm_ops.add_rmsnorm(x, d, w, 1e-5)
    for weight in (w[:512], w[:1], w.cpu()):
        with pytest.raises(ValueError):
            lm_ops.add_rmsnorm(x, x, weight, 1e-5)
        with pytest.raises(ValueError):
            lm_ops.RMSNormFunction.apply(x, weight, 1e-5)
    q, k = rnd(2, 9, 4, 32), rnd(2, 9, 2, 32)
    ct, st = lm_ops.rotary_tables_f32(*lm.rotary_tables(9, 32, 10000.0, q.device, torch.bfloat16))
    for args in ((q, k, ct[:8], st), (q, k, ct, st[:, :8]), (q, k[:, :8], ct, st), (q, k[:1], ct, st), (q, k.float(), ct, st), (q, k, ct.cpu(), st)):
        with pytest.raises(ValueError):
            lm_ops.rotary_pair(*args)
    norm = lm.RMSNorm(768, 1e-5).cuda().bfloat16()
    d = rnd(1, 6, 768)
    s, y = lm.add_norm(norm, x, d)
    assert torch.equal(s, x + d) and torch.equal(y, norm(x + d))
