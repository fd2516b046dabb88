"""A prompt through a patched block calls operators in place of torch modules: only where the modules would do
nothing else, whatever a program has changed about them since the last call."""

import copy

import pytest
import torch

from metile_b200 import backends
from metile_b200.integrations import blocks
from metile_b200.integrations.torch_lm import apply_metile_to_torch_lm, prompt_attention


def stand_in_projection(values, weight, scales, biases, *, group_size=64, bits=4):
    dense = (scales.float() * (1 + weight[:, ::8].view(torch.int32).float().abs() / 2**31)).repeat_interleave(64, dim=1)
    return torch.nn.functional.linear(values.float(), dense + biases.float().mean()).to(values.dtype) * (bits / 4)


def stand_in_norm(values, weight, eps):
    return (torch.nn.functional.rms_norm(values.float(), weight.shape, eps=eps) * weight.float()).to(values.dtype)


@pytest.fixture
def block(monkeypatch):
    monkeypatch.setattr(backends, "mlx_affine_qmv", stand_in_projection)
    monkeypatch.setattr(backends, "mlx_rms_norm", stand_in_norm)
    model = blocks.random_model(1, hidden=128, intermediate=128, heads=2, kv_heads=1, layers=1, vocab=64, device="cpu")
    # The patched norm asks for a CUDA device; here its own replacement is what a GPU would run.
    with apply_metile_to_torch_lm(model, attention=True):
        replacement = blocks.RMSNorm.forward
        norm_forward = lambda self, values: backends.mlx_rms_norm(values, self.weight, self.eps)  # noqa: E731
        norm_forward._metile_original = replacement._metile_original
        norm_forward._metile_replacement = norm_forward
        blocks.RMSNorm.forward = norm_forward
        yield model.layers[0]


def both_ways(block):
    values = torch.randn(1, 5, 128, generator=torch.Generator().manual_seed(7)).to(torch.bfloat16)

    def cache():
        return blocks.KVCache(1, 1, 8, 64, "cpu")
    short = prompt_attention(block.input_layernorm, block.self_attn, values, cache())
    return short, block.self_attn(block.input_layernorm(values), cache())


def doubled(forward):
    return lambda *args, **kwargs: 2 * forward(*args, **kwargs)


def test_the_modules_as_they_were_made(block):
    short, modules = both_ways(block)
    assert short is not None and torch.equal(short, modules)


@pytest.mark.parametrize("change", [
    lambda b: setattr(b.input_layernorm, "eps", 0.5),
    lambda b: setattr(b.self_attn, "scale", 0.01),
    lambda b: setattr(b.self_attn, "rope_theta", 1e2),
    lambda b: setattr(b.self_attn.q_proj, "scales", b.self_attn.q_proj.scales * 2),
    lambda b: setattr(b.self_attn, "o_proj", blocks.QuantizedLinear.from_seed(9, 128, 128)),
    lambda b: b.input_layernorm.weight.mul_(3),
])
def test_changed_tensors_and_settings_count(block, change):
    before, _ = both_ways(block)
    change(block)
    short, modules = both_ways(block)
    assert short is not None and torch.equal(short, modules) and not torch.equal(short, before)


@pytest.mark.parametrize("change", [
    lambda b: setattr(b.self_attn, "forward", doubled(b.self_attn.forward)),
    lambda b: setattr(b.self_attn.v_proj, "forward", doubled(b.self_attn.v_proj.forward)),
    lambda b: setattr(b.input_layernorm, "forward", doubled(b.input_layernorm.forward)),
    lambda b: setattr(b.self_attn.o_proj, "bias", torch.ones(128, dtype=torch.bfloat16)),
    lambda b: setattr(b.self_attn.o_proj, "bias", torch.nn.Parameter(torch.ones(128, dtype=torch.bfloat16))),
    lambda b: setattr(b.self_attn.v_proj, "bits", 8),
    lambda b: setattr(b.self_attn, "v_proj", torch.nn.Linear(128, 64, dtype=torch.bfloat16)),
    lambda b: setattr(b.input_layernorm, "weight", b.input_layernorm.weight.float()),
    lambda b: b.self_attn.v_proj.register_forward_hook(lambda module, args, out: 2 * out),
    lambda b: b.self_attn.register_forward_pre_hook(lambda module, args: (2 * args[0], args[1])),
    lambda b: b.self_attn.o_proj.register_full_backward_hook(lambda *args: None),
    lambda b: b.self_attn.o_proj.register_full_backward_pre_hook(lambda *args: None),
    lambda b: setattr(b.self_attn.k_proj, "_compiled_call_impl", b.self_attn.k_proj._call_impl),
])
def test_what_a_call_of_the_module_adds_is_not_left_out(block, change):
    assert both_ways(block)[0] is not None
    change(block)
    assert both_ways(block)[0] is None


def test_global_hooks_and_classes_changed_under_it(block, monkeypatch):
    handle = torch.nn.modules.module.register_module_forward_hook(lambda module, args, out: None)
    assert both_ways(block)[0] is None
    handle.remove()
    assert both_ways(block)[0] is not None
    for kind in (blocks.QuantizedLinear, blocks.Attention, blocks.RMSNorm):
        with monkeypatch.context() as patch:
            forward = doubled(kind.forward)
            forward.__dict__.update(kind.forward.__dict__)  # as functools.wraps would
            patch.setattr(kind, "forward", forward)
            assert both_ways(block)[0] is None
        with monkeypatch.context() as patch:
            patch.setattr(kind, "__call__", doubled(kind.__call__))
            assert both_ways(block)[0] is None
    assert both_ways(block)[0] is not None


def test_frequency_tables_belong_to_a_stream_and_not_to_the_module(block, monkeypatch):
    attention, cpu = block.self_attn, torch.device("cpu")
    stream, capturing = [1], [False]
    monkeypatch.setattr(blocks, "_current_stream", lambda device: stream[0])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    table = attention._frequencies_on(cpu)
    assert torch.equal(table, blocks._rope_frequencies(1e6, 64, cpu)) and attention._frequencies_on(cpu) is table
    stream[0] = 2
    assert attention._frequencies_on(cpu) is not table      # made in another stream's order
    stream[0] = 1
    assert attention._frequencies_on(cpu) is table
    capturing[0] = True
    assert attention._frequencies_on(cpu) is not table      # a graph may outlive what is kept
    capturing[0] = False
    attention.head_dim = 32
    assert attention._frequencies_on(cpu).shape == (16,)
    attention.head_dim = 64
    attention.rope_theta = 1e2
    assert torch.equal(attention._frequencies_on(cpu), blocks._rope_frequencies(1e2, 64, cpu))
    for stream[0] in range(3, 40):
        attention._frequencies_on(cpu)
        assert len(blocks._frequency_tables[attention]) <= 4
    # Nothing of it is saved or copied with the module.
    assert not any(isinstance(value, (torch.Tensor, tuple)) for value in vars(attention).values())
    assert copy.deepcopy(attention) not in blocks._frequency_tables


def test_a_cache_with_methods_of_its_own_is_not_passed_by(monkeypatch):
    cache = blocks.KVCache(1, 1, 8, 64, "cpu")
    assert blocks.appends_in_place(cache)
    for name in ("update_and_fetch", "advance"):
        other = blocks.KVCache(1, 1, 8, 64, "cpu")
        setattr(other, name, getattr(other, name))
        assert not blocks.appends_in_place(other)
        with monkeypatch.context() as patch:
            patch.setattr(blocks.KVCache, name, doubled(getattr(blocks.KVCache, name)))
            assert not blocks.appends_in_place(cache)

    class Counted(blocks.KVCache):
        pass
    assert not blocks.appends_in_place(Counted(1, 1, 8, 64, "cpu"))


def test_a_forward_that_tells_no_parameters_is_asked_for_all_logits():
    from metile_b200.integrations import graphed

    assert graphed._takes(blocks.TinyCausalLM.forward, "logits_to_keep")
    assert not graphed._takes(blocks.DecoderBlock.forward, "logits_to_keep")
    assert not graphed._takes(dict.fromkeys, "logits_to_keep") and not graphed._takes(type("C", (), {}).__new__, "x")
    assert not graphed._takes(max, "logits_to_keep")  # inspect.signature raises ValueError


def test_fused_projections_are_complete_before_they_are_kept(block, monkeypatch):
    from metile_b200.integrations import torch_lm

    class Stream:
        waits = 0

        def synchronize(self):
            assert block.self_attn not in torch_lm._qkv_cache
            Stream.waits += 1

    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    torch_lm._fused_qkv(block.self_attn)
    assert Stream.waits == 0 and block.self_attn not in torch_lm._qkv_cache
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    weight, scales, biases = torch_lm._fused_qkv(block.self_attn)
    assert Stream.waits == 1 and torch_lm._fused_qkv(block.self_attn)[0] is weight and Stream.waits == 1
    assert weight.shape[0] == scales.shape[0] == biases.shape[0] == 128 + 64 + 64
