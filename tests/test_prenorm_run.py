"""A model's layers launched by one native call against the same layers launched part by part."""
import pytest
import torch

from inferflux_b200 import Engine, StepEntry
from inferflux_b200.kernels import ops
from inferflux_b200.parts.feed_forward import SwiGLU

pytestmark = pytest.mark.gpu

CONFIG = dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", hidden_size=512, num_hidden_layers=3, num_attention_heads=4,
              num_key_value_heads=2, head_dim=128, intermediate_size=8192, vocab_size=1000, rope_theta=1e6, rms_norm_eps=1e-6,
              tie_word_embeddings=False, max_position_embeddings=8192, use_sliding_window=False, hidden_act="silu", torch_dtype="bfloat16")


def _run(native, steps, change=None, **config):
    engine = Engine.from_config(dict(CONFIG, **config), seed=3, dtype="bfloat16", kv_cache_tokens=16384, max_seqs=40, max_batch_size=40,
                                max_batch_tokens=8192, max_model_len=4096)
    model = engine.runner.model
    if change is not None:
        change(model)
    took = []
    if not native:
        model._prenorm_run = None
    elif model._prenorm_run is not None:
        forward = model._prenorm_run.forward
        model._prenorm_run.forward = lambda *a: (out := forward(*a), took.append(out is not None))[0]
    gen, out, counts = torch.Generator().manual_seed(5), [], []
    for step in steps:
        entries = []
        for rid, n in step:
            tokens = torch.randint(0, 1000, (n,), generator=gen).tolist()
            entries.append(StepEntry(rid, tokens, [0, n - 1] if n > 1 else [0]))
        before = ops.launch_count
        out.append(engine.run_step(entries).clone())
        counts.append(ops.launch_count - before)
    ops.check_device_errors("cuda:0")
    return out, counts, sum(took)


@pytest.mark.parametrize("steps,native_steps", [
    ([[("a", 9)], [("b", 16), ("a", 1)], [("c", 17)], [("d", 128)], [("e", 129)], [("f", 8)]], 4),         # the rows' edges
    ([[("a", 77)], [("a", 51)], [("b", 100), ("c", 28)]], 3),                                             # short prompts, several of them
    ([[("a", 900)], [("a", 60)], [("b", 1500), ("c", 40), ("d", 33)], [("a", 50), ("b", 1), ("c", 1)],    # portions behind a context, cut keys;
      [("a", 1), ("b", 20), ("c", 1), ("d", 1)]], 3),                                                     # single tokens of even and uneven contexts
])
def test_layers_of_one_call_are_the_parts_layers(steps, native_steps):
    """Bit for bit the same logits, as many kernels, and only steps of 9 to 128 rows with a portion among them."""
    want, want_counts, _ = _run(False, steps)
    got, counts, took = _run(True, steps)
    assert took == native_steps
    assert counts == want_counts
    for w, g in zip(want, got):
        assert torch.equal(w, g)


STEPS = [[("a", 9)], [("a", 16)], [("b", 17), ("a", 1)], [("c", 900)], [("c", 77), ("a", 1)], [("d", 128)], [("c", 40), ("b", 1), ("d", 3)]]


@pytest.mark.parametrize("config", [dict(hidden_size=768, num_attention_heads=6, num_key_value_heads=6, intermediate_size=8200),
                                    dict(hidden_size=1032, num_attention_heads=16, num_key_value_heads=2, num_hidden_layers=2, intermediate_size=11008)])
def test_layers_of_other_sizes(config):
    """Other widths and numbers of heads, at the rows where the kernels change."""
    want, want_counts, _ = _run(False, STEPS, **config)
    got, counts, took = _run(True, STEPS, **config)
    assert took == 6 and counts == want_counts
    for w, g in zip(want, got):
        assert torch.equal(w, g)


def _off_the_boundary(model):
    linear = model.blocks[1].mixer.o
    room = torch.empty(linear.weight.numel() + 1, dtype=torch.bfloat16, device=linear.weight.device)
    linear.weight = room[1:].view(linear.weight.shape).copy_(linear.weight)


def _half_the_rotation(model):
    (position,) = model.positions.values()
    position.rotary_dim, position.inv_freq = 64, position.inv_freq[:32].contiguous()


def _float32_weights(model):
    linear = model.blocks[2].feed_forward.down
    linear.weight = linear.weight.float()


def _biased(model):
    linear = model.blocks[0].mixer.o
    linear.bias = torch.randn(linear.out_features, generator=torch.Generator().manual_seed(2)).to(linear.weight.device)


@pytest.mark.parametrize("change", [_off_the_boundary, _half_the_rotation, _float32_weights, _biased])
def test_what_the_call_does_not_take_goes_through_the_blocks(change):
    """Weights off the 16-byte boundaries, of another type or with a bias, another width of the rotation: nothing of the call has been
    done, and the blocks' results come out."""
    want, want_counts, _ = _run(False, STEPS, change)
    got, counts, took = _run(True, STEPS, change)
    assert took == 0 and counts == want_counts
    for w, g in zip(want, got):
        assert torch.equal(w, g)


def test_models_of_another_kind_keep_their_blocks():
    from inferflux_b200.engine.prenorm_run import PrenormRun
    for other in (dict(head_dim=64), dict(intermediate_size=1024), dict(use_sliding_window=True, sliding_window=64, max_window_layers=0)):
        engine = Engine.from_config(dict(CONFIG, **other), seed=3, dtype="bfloat16", kv_cache_tokens=1024, max_seqs=2, max_model_len=512)
        assert PrenormRun.of(engine.runner.model) is None


WATCHED = {
    "block": lambda m: m.blocks[1], "mixer": lambda m: m.blocks[2].mixer, "norm": lambda m: m.blocks[0].mixer_norm,
    "second norm": lambda m: m.blocks[1].feed_forward_norm, "feed-forward": lambda m: m.blocks[1].feed_forward,
    "qkv": lambda m: m.blocks[0].mixer.qkv, "down": lambda m: m.blocks[2].feed_forward.down}


@pytest.mark.parametrize("of_the_class", [False, True])
@pytest.mark.parametrize("what", sorted(WATCHED))
def test_a_method_put_on_a_part_is_called(what, of_the_class, monkeypatch):
    """A forward that stands on a block or part, or on its class, is called in these steps like in others; when it is gone, one call again."""
    engine = Engine.from_config(CONFIG, seed=3, dtype="bfloat16", kv_cache_tokens=4096, max_seqs=4, max_model_len=512)
    model = engine.runner.model
    part, seen, took = WATCHED[what](model), [], []
    forward = model._prenorm_run.forward
    model._prenorm_run.forward = lambda *a: took.append(1) or forward(*a)
    tokens = torch.randint(0, 1000, (40,), generator=torch.Generator().manual_seed(1)).tolist()
    want = engine.run_step([StepEntry("a", tokens, [0, 39])]).clone()
    assert len(took) == 1
    with monkeypatch.context() as patch:
        if of_the_class:
            inner = type(part).forward
            patch.setattr(type(part), "forward", lambda self, *a, **k: (seen.append(self is part), inner(self, *a, **k))[1])
        else:
            inner = part.forward
            patch.setattr(part, "forward", lambda *a, **k: (seen.append(True), inner(*a, **k))[1], raising=False)
        got = engine.run_step([StepEntry("b", tokens, [0, 39])]).clone()
        assert any(seen) and len(took) == 1
    part.__dict__.pop("forward", None)
    assert torch.equal(got, want) and torch.equal(engine.run_step([StepEntry("c", tokens, [0, 39])]), want)
    assert len(took) == 2


def test_a_part_put_in_anothers_place_is_called():
    class Watched(SwiGLU):
        calls = 0

        def forward(self, x, ctx):
            Watched.calls += 1
            return super().forward(x, ctx)
    engine = Engine.from_config(CONFIG, seed=3, dtype="bfloat16", kv_cache_tokens=4096, max_seqs=4, max_model_len=512)
    model = engine.runner.model
    block = model.blocks[1]
    made = block.feed_forward
    other = Watched.__new__(Watched)
    other.__dict__.update(made.__dict__)
    block.feed_forward = other
    engine.run_step([StepEntry("a", list(range(40)), [39])])
    assert Watched.calls == 1
    block.feed_forward = made
    model.blocks[1] = type("Block", (), {"forward": lambda self, *a: (setattr(Watched, "calls", 5), block.forward(*a))[1]})()
    engine.run_step([StepEntry("b", list(range(40)), [39])])
    assert Watched.calls == 5
