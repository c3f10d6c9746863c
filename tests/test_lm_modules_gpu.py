"""GPU: norms and projections of the LM that are hooked, wrapped or replaced take part in the forward pass, which takes the plain ones'
steps in joined native calls."""
import pytest
import torch
import torch.nn.functional as F

from oracle import mhffn_oracle as orc

pytestmark = pytest.mark.gpu


def _model():
    from flashmhf_b200 import lm
    cfg = lm.LMConfig(vocab_size=97, hidden_size=768, num_hidden_layers=2, num_attention_heads=12, num_key_value_heads=12, intermediate_size=128,
                      mhffnmoe_num_heads=8, mhffnmoe_num_kuv_heads=8, mhffnmoe_num_experts=2, mhffnmoe_apply_rmsnorm=False)
    m = lm.DecoderLM(cfg).cuda().bfloat16().init_weights(seed=1)
    return m, torch.randint(0, 97, (2, 40), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))


class _Shifted(torch.nn.Module):
    """Another norm in the place of an RMSNorm, with the same attributes."""

    def __init__(self, norm):
        super().__init__()
        self.weight, self.eps = norm.weight, norm.eps

    def forward(self, x):
        return F.layer_norm(x, (x.shape[-1],), self.weight, None, self.eps) + 1


@pytest.mark.parametrize("grad", [False, True])
def test_norms(grad):
    m, ids = _model()
    with torch.set_grad_enabled(grad):
        want, seen = m(ids), []
        norms = [m.model.layers[0].post_attention_layernorm, m.model.layers[1].input_layernorm, m.model.norm]
        hooks = [n.register_forward_hook(lambda mod, a, out: seen.append(mod)) for n in norms]
        assert orc.rel_l2(m(ids), want) < 2e-2 and seen == norms
        for h in hooks:
            h.remove()
        m.model.norm = _Shifted(m.model.norm)
        shifted = m(ids)
        m.model.norm, last = torch.nn.Identity(), m.model.norm
        assert orc.rel_l2(shifted, m.lm_head(last(m.hidden(ids)))) < 2e-2


class _LowRank(torch.nn.Module):
    """A projection with an addition of its own, as an adapter puts it in place."""

    def __init__(self, lin):
        super().__init__()
        self.base, self.weight = lin, lin.weight
        self.down = torch.nn.Parameter(torch.full((4, lin.in_features), 0.02, device="cuda", dtype=torch.bfloat16))
        self.up = torch.nn.Parameter(torch.full((lin.out_features, 4), 0.05, device="cuda", dtype=torch.bfloat16))

    def forward(self, x):
        return self.base(x) + F.linear(F.linear(x, self.down), self.up)


@pytest.mark.parametrize("name", ["q_proj", "k_proj", "v_proj", "o_proj"])
def test_projections(name):
    m, ids = _model()
    att = m.model.layers[0].self_attn
    with torch.no_grad():
        plain, seen = m(ids), []
        h = getattr(att, name).register_forward_hook(lambda mod, a, out: seen.append(out.shape))
        assert orc.rel_l2(m(ids), plain) < 2e-2 and len(seen) == 1
        h.remove()
        setattr(att, name, _LowRank(getattr(att, name)))
        got = m(ids)
        lin = getattr(att, name)
        bias = torch.nn.Linear(768, 768, device="cuda", dtype=torch.bfloat16)
        bias.weight.copy_(lin.weight)
        bias.bias.fill_(0.5)
        setattr(att, name, bias)
        biased = m(ids)
    with torch.enable_grad():        # every module is called here
        setattr(att, name, lin)
        assert orc.rel_l2(got, m(ids).detach()) < 2e-2
        setattr(att, name, bias)
        assert orc.rel_l2(biased, m(ids).detach()) < 2e-2
