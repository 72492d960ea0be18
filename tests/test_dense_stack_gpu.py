"""A dense decoder's layers from one native call against the same layers part by part."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(dtype, heads, kv_heads, dim, hidden, inter, layers, page, tied=True):
    from tinyinfer_b200.config import Qwen3Config
    from tinyinfer_b200 import models  # noqa: F401
    from tinyinfer_b200.config import lookup_architecture
    cfg = dict(architectures=["Qwen3ForCausalLM"], vocab_size=515, hidden_size=hidden, num_hidden_layers=layers, num_attention_heads=heads,
               num_key_value_heads=kv_heads, head_dim=dim, intermediate_size=inter, rms_norm_eps=1e-6, rope_theta=1e6,
               tie_word_embeddings=tied, max_position_embeddings=4096)
    arch = lookup_architecture("Qwen3ForCausalLM")
    return fill(arch.model_factory(Qwen3Config.from_dict(cfg), dtype, torch.device("cuda:0")), dtype, page)


def fill(model, dtype, page):
    """The model with random weights, and what makes runners of it."""
    from tinyinfer_b200.engine.runner import ModelRunner
    gen = torch.Generator(device="cuda:0").manual_seed(3)
    tensors = {}
    for name, ts in model.expected_tensors().items():
        t = torch.randn(tuple(ts.shape), generator=gen, device="cuda:0")
        tensors[name] = 1.0 + 0.1 * t if ts.role == "vector32" else (t * (1.0 if "embed" in name else 0.05)).to(dtype)
    model.load_tensors(tensors)
    return model, lambda graphs=False: ModelRunner(model, page_size=page, num_pages=900, max_requests=12, max_tokens_per_step=3000,
                                                   max_model_len=2600, cuda_graphs=graphs)


STEPS = [[(0, 37)], [(8, 8)], [(9, 3)], [(0, 1)], [(0, 1), (1, 300)], [(0, 1), (1, 1), (2, 64), (3, 65)], [(4, 2200)], [(4, 130), (0, 1), (5, 9)],
         [(i, 1) for i in range(6)], [(4, 1), (6, 7)], [(i, 1) for i in range(7)] + [(7, 600)]]


def run(runner, steps):
    from tinyinfer_b200.engine.batch import StepEntry
    gen = torch.Generator().manual_seed(5)
    return [runner.step([StepEntry(r, torch.randint(0, 515, (n,), generator=gen).tolist(), [0, n - 1] if n > 1 else [0])
                         for r, n in step]).clone() for step in steps]


@pytest.mark.parametrize("dtype,heads,kv_heads,dim,hidden,inter,page", [
    (torch.bfloat16, 4, 2, 64, 256, 384, 16), (torch.bfloat16, 8, 1, 128, 520, 1000, 64), (torch.float32, 4, 2, 128, 256, 320, 64),
    (torch.float32, 6, 2, 64, 260, 328, 5)])
def test_stack_equals_the_parts(dtype, heads, kv_heads, dim, hidden, inter, page):
    from tinyinfer_b200 import ops
    model, runner = make(dtype, heads, kv_heads, dim, hidden, inter, 3, page)
    stack = model._stack
    assert stack is not None
    # the kernels are the parts', on the same operands in the same order: so are the bits
    for graphs in (False, True):
        model._stack = None
        want = run(runner(graphs), STEPS)
        model._stack = stack
        got = run(runner(graphs), STEPS)
        for g, w, step in zip(got, want, STEPS):
            assert torch.isfinite(g).all() and torch.equal(g, w), (step, ((g - w).norm() / w.norm()).item())
    ops.check_kernel_status()


def test_what_the_stack_does_not_take(monkeypatch):
    """Sizes of other kernels run part by part."""
    from tinyinfer_b200 import ops
    called = []
    real = ops.dense_stack
    monkeypatch.setattr(ops, "dense_stack", lambda *a, **k: called.append(1) or real(*a, **k))
    for dtype, heads, kv, dim, hidden, inter, page, taken in (
            (torch.bfloat16, 4, 2, 32, 128, 256, 16, False), (torch.bfloat16, 4, 2, 64, 132, 256, 16, False),
            (torch.bfloat16, 4, 2, 64, 128, 256, 8, False), (torch.bfloat16, 4, 2, 64, 128, 256, 16, True),
            (torch.float32, 4, 2, 48, 128, 256, 16, False)):
        _, runner = make(dtype, heads, kv, dim, hidden, inter, 2, page)
        del called[:]
        out = run(runner(), [[(0, 20)], [(0, 1)]])
        assert bool(called) == taken and all(torch.isfinite(o).all() for o in out)


@pytest.mark.parametrize("heads,kv_heads,dim", [(5, 1, 128), (3, 3, 64), (7, 1, 64), (12, 4, 128)])
def test_portions_beside_decoded_tokens_behind_a_long_prefix(heads, kv_heads, dim):
    """Odd numbers of heads and rows: where the portions' keys are shared out over CTAs, their partial results lie behind the
    decoded tokens' on one scratch. The kernels are the parts', and so are the bits."""
    from tinyinfer_b200 import ops
    model, runner = make(torch.bfloat16, heads, kv_heads, dim, 64 * heads, 384, 2, 64)
    steps = [[(0, 2300)], [(1, 40), (2, 33), (3, 21)], [(1, 1), (0, 40)], [(2, 1), (0, 60), (1, 1)], [(1, 1), (2, 1), (3, 1), (0, 130)]]
    got = run(runner(), steps)
    model._stack = None
    want = run(runner(), steps)
    assert all(torch.equal(g, w) and torch.isfinite(g).all() for g, w in zip(got, want))
    ops.check_kernel_status()


def make_mixed(dtype, table, page=16):
    """Layers with and without a window, one that runs twice, an entry that only reads what another cached; with ``table``
    also biases, norms of q and k, gelu, and a rotation of neighbouring features by a table, else positions are not used."""
    from tinyinfer_b200 import ops
    from tinyinfer_b200.config import AttentionSpec, ExecStep, GatedMLPSpec, LayerSpec, ModelSpec, NormSpec, PositionSpec
    from tinyinfer_b200.models import DecoderModel
    norm = NormSpec(256, 1e-5)

    def layer(window):
        mixer = AttentionSpec(hidden_size=256, num_heads=6, num_kv_heads=2, head_dim=64, scale=0.11, position=PositionSpec(kind="none"),
                              qk_norm=NormSpec(64, 1e-4) if table else None, bias=table, window=window)
        return LayerSpec(mixer=mixer, feed_forward=GatedMLPSpec(256, 384, activation="gelu_tanh" if table else "silu"),
                         mixer_norm=norm, feed_forward_norm=norm)
    spec = ModelSpec(architecture="Mixed", vocab_size=515, hidden_size=256, layers=(layer(40), layer(None), layer(300)),
                     execution=(ExecStep(0, 0), ExecStep(1, 1), ExecStep(1, 2), ExecStep(2, 3), ExecStep(2, 3, writes_cache=False),
                                ExecStep(0, 4)),
                     final_norm=norm, tie_embeddings=True, max_positions=4096)
    model = DecoderModel(spec, dtype, "cuda:0")
    if table:
        angle = torch.log1p(torch.arange(4096.0))[:, None] * 100.0 ** (-torch.arange(24.0) / 24)
        turn = ops.Rotation(48, cos_sin=torch.cat([angle.cos(), angle.sin()], dim=1).contiguous().cuda(), interleaved=True)
        for b in model.blocks:
            b.mixer._rotation = turn
    return fill(model, dtype, page)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("table", [False, True])
def test_stack_of_windows_biases_tables_and_shared_entries(dtype, table):
    """Everything that a layer can hand to the native call, bit for bit as the parts run it, and the same bits every time."""
    from tinyinfer_b200 import ops
    model, runner = make_mixed(dtype, table)
    stack = model._stack
    assert stack is not None
    taken = []
    run_stack = stack.run
    stack.run = lambda x, step: taken.append(run_stack(x, step)) or taken[-1]
    for graphs in (False, True):
        model._stack = None
        want = run(runner(graphs), STEPS)
        model._stack = stack
        for _ in range(3):
            got = run(runner(graphs), STEPS)
            for g, w, step in zip(got, want, STEPS):
                assert torch.isfinite(g).all() and torch.equal(g, w), (step, ((g - w).norm() / w.norm()).item())
    assert taken and all(t is not None for t in taken)
    ops.check_kernel_status()
