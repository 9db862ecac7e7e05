"""Which decode steps the model hands to the one-launch step, and what with.  The launch itself is replaced: no GPU needed."""
import pytest
import torch


@pytest.fixture
def step(pkg, monkeypatch):
    """A small model of stock layers, and a function that runs the decision for a decode step: what ops.decode_stack was called
    with, or None where the layers would run one by one."""
    from nanovllm_b200 import ops
    from nanovllm_b200.engine.model_runner import ModelConfig
    from nanovllm_b200.models.qwen3 import Qwen3Model
    from nanovllm_b200.utils.context import reset_context, set_context
    model = Qwen3Model(ModelConfig(hidden_size=64, num_attention_heads=2, num_key_value_heads=1, head_dim=32, intermediate_size=64, num_hidden_layers=3, vocab_size=16,
                                   max_position_embeddings=64))
    for layer in model.layers:
        layer.self_attn.attn.k_cache = layer.self_attn.attn.v_cache = torch.zeros(2, 16, 1, 32)
    calls = []
    monkeypatch.setattr(ops, "decode_stack", lambda *a: calls.append(a) or ("normed" if a[2] else None))
    monkeypatch.setattr(ops, "decode_stack_served", lambda rows, *shape: shape == (3, 64, 2, 1, 32, 64, 16) and rows <= 16)

    def run(rows=2):
        calls.clear()
        ints = torch.ones(rows, dtype=torch.int32)
        set_context(False, slot_mapping=ints, context_lens=ints, block_tables=ints.view(-1, 1))
        try:
            out = model._decode_in_one_launch(torch.zeros(rows, 64), torch.zeros(rows, dtype=torch.int64))
        finally:
            reset_context()
        assert (out == "normed") == (len(calls) == 1 and len(calls[0][2]) > 0)
        return None if out is None else calls[0]

    run.model = model
    return run


def test_stock_layers_go_in_one_launch(step):
    call = step()
    assert len(call[2]) == 3 and call[10] == 32 ** -0.5


def test_scale_of_a_single_layer(step):
    """The launch takes one scale of attention for all layers."""
    attns = [layer.self_attn.attn for layer in step.model.layers]
    attns[1].scale *= 2
    assert step() is None
    attns[0].scale *= 2
    attns[2].scale *= 2
    assert step()[10] == 2 * 32 ** -0.5


def test_nothing_is_gathered_for_a_step_that_is_not_served(step, monkeypatch):
    from nanovllm_b200.models import qwen3
    asked = []
    stock = qwen3._is_stock
    monkeypatch.setattr(qwen3, "_is_stock", lambda layer: asked.append(layer) or stock(layer))
    assert step(17) is None and len(asked) <= 1
    assert step(16) is not None and len(asked) > 3


def test_first_layer_of_another_kind(step):
    step.model.layers[0] = torch.nn.Identity()
    assert step() is None


def _ignore(*_):
    return None


@pytest.mark.parametrize("register", ["register_module_forward_pre_hook", "register_module_forward_hook", "register_module_full_backward_pre_hook",
                                      "register_module_full_backward_hook"])
def test_hooks_for_all_modules(step, register):
    handle = getattr(torch.nn.modules.module, register)(_ignore)
    try:
        assert step() is None
    finally:
        handle.remove()
    assert step() is not None


@pytest.mark.parametrize("register", ["register_forward_pre_hook", "register_forward_hook", "register_full_backward_pre_hook", "register_full_backward_hook"])
@pytest.mark.parametrize("where", ["layers.1", "layers.0.input_layernorm"])
def test_hooks_of_a_module(step, register, where):
    handle = getattr(step.model.get_submodule(where), register)(_ignore)
    assert step() is None
    handle.remove()
    assert step() is not None


METHODS = [("layers.1", "forward"), ("layers.0.input_layernorm", "forward"), ("layers.0.input_layernorm", "rms_forward"), ("layers.2.self_attn", "attention_output"),
           ("layers.2.self_attn.attn", "attend"), ("layers.1.self_attn.o_proj", "forward_fused"), ("layers.1.mlp", "activation"),
           ("layers.1.mlp.gate_up_proj", "forward_silu_mul"), ("layers.1.mlp.gate_up_proj", "paired_weight"), ("layers.1.mlp.down_proj", "forward_fused")]


@pytest.mark.parametrize("where,name", METHODS)
@pytest.mark.parametrize("of", ["object", "class"])
def test_replaced_methods(step, monkeypatch, where, name, of):
    module = step.model.get_submodule(where)
    method = getattr(type(module), name)
    with monkeypatch.context() as m:
        if of == "object":
            module.__dict__[name] = lambda *a: method(module, *a)
        else:
            m.setattr(type(module), name, lambda self, *a: method(self, *a))
        assert step() is None
    module.__dict__.pop(name, None)
    assert step() is not None


@pytest.mark.parametrize("where", ["layers.1", "layers.0.input_layernorm"])
def test_modules_compiled_in_place(step, where):
    step.model.get_submodule(where).compile(backend="eager")
    assert step() is None
