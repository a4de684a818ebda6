"""Decoder blocks call their attention and norm modules where someone hooks, overrides or replaces them, and give the
same result whichever way they run."""
import pytest
import torch
import torch.nn as nn

from merak_b200.models.gpt2 import GPT2Attention, GPT2Block, GPT2LMHeadModel, gpt2_config
from merak_b200.models.llama import LlamaDecoderLayer, llama_config
from merak_b200.models.moe import MoEDecoderLayer, deepseek_v2_config
from merak_b200.ops.rng import dropout_state
from merak_b200.pipeline.profiler import FlopsProfiler


def _gpt2_block(p=0.3):
    torch.manual_seed(0)
    return GPT2Block(gpt2_config("gpt2", n_embd=64, n_head=1, resid_pdrop=p, attn_pdrop=0.0))


def _run(block, x, call=7):
    dropout_state().set_call_id(call)
    return block(x)


def _llama():
    torch.manual_seed(0)
    return LlamaDecoderLayer(llama_config("llama-tiny"))


def _moe():
    torch.manual_seed(0)
    return MoEDecoderLayer(deepseek_v2_config("deepseek-v2-lite", hidden_size=64, num_attention_heads=2, intermediate_size=64,
                                              n_routed_experts=0), 0)


@pytest.mark.parametrize("train", [True, False])
@pytest.mark.parametrize("which", ["ln_1", "attn", "ln_2", "mlp"])
def test_hooks_fire_in_both_modes(train, which):
    block, x = _gpt2_block().train(train), torch.randn(2, 5, 64)
    want = _run(block, x)
    seen = []
    getattr(block, which).register_forward_hook(lambda m, args, out: seen.append(out))
    assert torch.allclose(_run(block, x), want, atol=1e-6)
    assert len(seen) == 1 and isinstance(seen[0], torch.Tensor) and seen[0].shape == x.shape


def test_attention_hook_sees_dropout_and_residual():
    """What the attention module returns in training does not depend on who asks."""
    block, x = _gpt2_block().train(), torch.randn(2, 5, 64)
    seen = []
    block.attn.register_forward_hook(lambda m, args, out: seen.append(out))
    _run(block, x)
    dropout_state().set_call_id(7)
    assert torch.equal(seen[0], block.attn(block.ln_1(x), x))


@pytest.mark.parametrize("how", ["subclass", "instance", "class", "global"])
def test_overridden_attention_is_called(how, monkeypatch):
    block, x = _gpt2_block().train(), torch.randn(2, 5, 64)
    calls = []

    def forward(self, n, residual=None):
        calls.append(1)
        return residual

    handle = None
    if how == "subclass":
        block.attn.__class__ = type("Other", (GPT2Attention,), {"forward": forward})
    elif how == "instance":
        block.attn.forward = lambda n, residual=None: forward(block.attn, n, residual)
    elif how == "class":
        monkeypatch.setattr(GPT2Attention, "forward", forward)
    else:
        handle = nn.modules.module.register_module_forward_hook(
            lambda m, args, out: calls.append(1) if m is block.attn else None)
    try:
        _run(block, x)
    finally:
        if handle is not None:
            handle.remove()
    assert calls == [1]


@pytest.mark.parametrize("make,norms", [(_gpt2_block, ("ln_1", "ln_2")),
                                        (_llama, ("input_layernorm", "post_attention_layernorm")),
                                        (_moe, ("input_layernorm", "post_attention_layernorm"))])
def test_replaced_norms(make, norms):
    """Any module that maps a tensor to a tensor can stand in for a norm, and a norm's hooks see tensors."""
    block = make().train()
    x = torch.randn(1, 4, getattr(block, norms[0]).weight.shape[0])
    for name in norms:
        seen = []
        getattr(block, name).register_forward_hook(lambda m, args, out: seen.append(out))
        _run(block, x)
        assert all(isinstance(o, torch.Tensor) for o in seen) and len(seen) == 1
        setattr(block, name, nn.Identity())
    assert _run(block, x).shape == x.shape


def test_dropout_does_not_follow_the_norms_mode():
    """A frozen norm in evaluation mode leaves the attention's dropout on."""
    block, x = _gpt2_block().train(), torch.randn(2, 5, 64)
    want = _run(block, x)
    block.ln_2.eval()
    assert torch.allclose(_run(block, x), want, atol=1e-6)


def test_profiler_counts_attention_of_a_training_step():
    torch.manual_seed(0)
    model = GPT2LMHeadModel(gpt2_config("gpt2", n_layer=2, n_embd=64, n_head=1, vocab_size=97)).train()
    prof = FlopsProfiler(model)
    prof.start_profile()
    model(torch.randint(0, 97, (1, 6)))
    prof.stop_profile()
    attention = [m for m in model.modules() if isinstance(m, GPT2Attention)]
    assert len(attention) == 2 and all(prof.flops.get(m, 0) > 0 and prof.latency.get(m, 0) > 0 for m in attention)
    prof.end_profile()
