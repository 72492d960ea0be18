"""Operands that are not as the kernels read them: the native call leaves them to the parts, whose calls refuse them."""
from types import SimpleNamespace

import pytest
import torch

from tinyinfer_b200 import models, ops  # noqa: F401  (registers the architectures)
from tinyinfer_b200.config import Qwen3Config, lookup_architecture


class Seeming(torch.Tensor):
    """A CPU tensor that says it is on the GPU."""
    is_cuda = True


def seeming(t):
    return t.as_subclass(Seeming)


def on_cpu(t):
    return t.as_subclass(torch.Tensor)


@pytest.fixture
def stack_and_step(monkeypatch):
    cfg = dict(architectures=["Qwen3ForCausalLM"], vocab_size=64, hidden_size=64, num_hidden_layers=2, num_attention_heads=2,
               num_key_value_heads=1, head_dim=64, intermediate_size=48, rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=True,
               max_position_embeddings=64)
    model = lookup_architecture("Qwen3ForCausalLM").model_factory(Qwen3Config.from_dict(cfg), torch.float32, torch.device("cpu"))
    model.load_tensors({n: torch.ones(tuple(t.shape)) for n, t in model.expected_tensors().items()})
    for b in model.blocks:
        for part in (b.mixer, b.feed_forward, b.mixer_norm, b.feed_forward_norm, b.mixer._rotation):
            for name, t in vars(part).items():
                if isinstance(t, torch.Tensor):
                    setattr(part, name, seeming(t))
    views = [SimpleNamespace(kv=seeming(torch.zeros(2, 3, 1, 16, 64)), block_table=seeming(torch.zeros(1, 4, dtype=torch.int32)), writes=True)
             for _ in range(2)]
    step = SimpleNamespace(positions=seeming(torch.zeros(5, dtype=torch.int32)), token_seq=seeming(torch.zeros(5, dtype=torch.int32)),
                           cache_view=lambda entry: views[entry.cache], views=views)
    monkeypatch.setattr(ops, "dense_stack", lambda *a, **k: "native")
    return model._stack, step


def run(stack, step):
    return stack.run(seeming(torch.zeros(5, 64)), step)


def test_the_call_is_made(stack_and_step):
    stack, step = stack_and_step
    assert run(stack, step) == "native"
    assert stack.run(torch.zeros(5, 64), step) is None and stack.run(seeming(torch.zeros(5, 32)), step) is None


PARTS = [("mixer", n) for n in ("w_qkv", "w_o", "q_norm", "k_norm")] + [("feed_forward", "w_gate_up"), ("feed_forward", "w_down"),
                                                                      ("mixer_norm", "weight"), ("feed_forward_norm", "weight")]
CHANGES = {
    "type": lambda t: seeming(on_cpu(t).to(torch.float64 if t.is_floating_point() else torch.int64)),
    "device": on_cpu,
    "gaps": lambda t: seeming(torch.zeros(*t.shape[:-1], 2 * t.shape[-1], dtype=t.dtype)[..., ::2]),
    "sizes": lambda t: seeming(torch.zeros(*t.shape[:-1], t.shape[-1] - 4, dtype=t.dtype)),
}


@pytest.mark.parametrize("change", CHANGES)
def test_weights_that_do_not_lie_as_they_are_read(stack_and_step, change):
    stack, step = stack_and_step
    for part, name in PARTS:
        holder = getattr(stack.blocks[1], part)
        right = getattr(holder, name)
        setattr(holder, name, CHANGES[change](right))
        assert run(stack, step) is None, (part, name)
        setattr(holder, name, right)
    for name, size in (("b_qkv", 256), ("b_o", 64)):
        setattr(stack.blocks[0].mixer, name, CHANGES[change](seeming(torch.zeros(size))))
        assert run(stack, step) is None, name
        setattr(stack.blocks[0].mixer, name, None)
    assert run(stack, step) == "native"


@pytest.mark.parametrize("change", ["type", "device", "gaps"])
def test_a_step_that_does_not_lie_as_it_is_read(stack_and_step, change):
    stack, step = stack_and_step
    for holder, name in [(step, "positions"), (step, "token_seq"), (step.views[1], "kv"), (step.views[1], "block_table")]:
        right = getattr(holder, name)
        setattr(holder, name, CHANGES[change](right))
        assert run(stack, step) is None, name
        setattr(holder, name, right)
    step.views[1].kv = seeming(torch.zeros(2, 3, 1, 8, 64))         # pages of another size than the first layer's
    assert run(stack, step) is None
