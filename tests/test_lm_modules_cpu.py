"""CPU: what a user puts around or in place of a decoder layer of the LM is called: hooks, wrappers, a replaced forward."""
import torch
from torch.distributed.algorithms._checkpoint.checkpoint_wrapper import checkpoint_wrapper

from flashmhf_b200 import lm
from tests.test_lm_cpu import tiny_model


class _Counted(torch.nn.Module):
    def __init__(self, inner):
        super().__init__()
        self.inner, self.calls = inner, 0

    def forward(self, *a, **kw):
        self.calls += 1
        return self.inner(*a, **kw)


def test_decoder_layers_are_called_where_they_are_more_than_themselves():
    m, ids = tiny_model()
    want = m(ids)
    seen = []
    h = m.model.layers[0].register_forward_hook(lambda mod, args, out: seen.append(out.shape))
    assert torch.equal(m(ids), want) and seen == [(2, 24, 128)]
    h.remove()
    h = m.model.layers[1].register_forward_pre_hook(lambda mod, args: (torch.zeros_like(args[0]), *args[1:]))
    assert not torch.equal(m(ids), want)
    h.remove()
    m.model.layers[1] = _Counted(m.model.layers[1])
    assert torch.equal(m(ids), want) and m.model.layers[1].calls == 1
    m.model.layers[1] = m.model.layers[1].inner
    inner = m.model.layers[0].forward
    m.model.layers[0].forward = lambda *a: 2 * inner(*a)
    assert not torch.equal(m(ids), want)
    del m.model.layers[0].forward
    every = torch.nn.modules.module.register_module_forward_hook(
        lambda mod, args, out: seen.append("layer") if isinstance(mod, lm.DecoderLayer) else None)
    assert torch.equal(m(ids), want) and seen.count("layer") == 2
    every.remove()


def test_checkpointed_layers_give_the_same_gradients():
    m, ids = tiny_model()
    m.loss(ids).backward()
    want = {n: p.grad.clone() for n, p in m.named_parameters()}
    m.zero_grad()
    for i in range(len(m.model.layers)):
        m.model.layers[i] = checkpoint_wrapper(m.model.layers[i])
    m.loss(ids).backward()
    for n, p in m.named_parameters():
        assert torch.equal(p.grad, want[n.replace("_checkpoint_wrapped_module.", "")]), n
