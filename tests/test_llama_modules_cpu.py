"""Which modules of a Llama layer are called: hooks, adapters and forwards of single objects take part in the projections."""
from types import SimpleNamespace

import pytest
import torch

CFG = SimpleNamespace(hidden_size=32, intermediate_size=64, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2, vocab_size=16,
                      max_position_embeddings=32, rope_theta=1e4, rms_norm_eps=1e-5, rope_scaling=None)


class Adapter(torch.nn.Module):
    def __init__(self, base):
        super().__init__()
        self.base = base

    def forward(self, x):
        return self.base(x) + 1


@pytest.mark.parametrize("name", ["q_proj", "k_proj", "v_proj"])
def test_projections_are_called(name):
    from pace_b200.llm.models.llama import LlamaForCausalLM
    at = LlamaForCausalLM(CFG).model.layers[0].self_attn
    x, i = torch.randn(5, 32), ("q_proj", "k_proj", "v_proj").index(name)
    want = at.project(x)[i]
    seen = []
    m = getattr(at, name)
    m.register_forward_hook(lambda *a: seen.append(1))
    assert torch.equal(at.project(x)[i], want) and seen == [1]
    setattr(at, name, Adapter(m))                     # has no weight of its own
    assert torch.equal(at.project(x)[i], want + 1)


def test_what_counts_as_untouched():
    from pace_b200.llm.models.llama import LlamaForCausalLM, RMSNorm, _untouched
    lay = LlamaForCausalLM(CFG).model.layers[0]
    norm = lay.input_layernorm
    assert lay.plain and _untouched(norm, RMSNorm)
    for register in ("register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook", "register_full_backward_pre_hook"):
        hook = getattr(norm, register)(lambda *a: None)
        assert not _untouched(norm, RMSNorm), register
        hook.remove()
    with torch.nn.modules.module.register_module_forward_pre_hook(lambda *a: None):
        assert not _untouched(norm, RMSNorm) and not lay.plain
    norm.forward = norm.forward
    assert not _untouched(norm, RMSNorm)
    del norm.forward
    assert _untouched(norm, RMSNorm)
    assert not _untouched(torch.nn.LayerNorm(4), RMSNorm)


def test_replaced_blocks_keep_their_weights_where_they_are():
    from pace_b200.llm.models.llama import LlamaForCausalLM
    model = LlamaForCausalLM(CFG)
    model.model.layers[0].self_attn = torch.nn.Linear(4, 4)        # no projections of its own
    model.model.layers[0].mlp = torch.nn.Identity()
    model.to(torch.float64)
