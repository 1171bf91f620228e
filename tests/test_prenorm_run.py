"""A model's layers launched by one native call against the same layers launched part by part."""
import pytest
import torch

from inferflux_b200 import Engine, StepEntry
from inferflux_b200.kernels import ops

pytestmark = pytest.mark.gpu

CONFIG = dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", hidden_size=512, num_hidden_layers=3, num_attention_heads=4,
              num_key_value_heads=2, head_dim=128, intermediate_size=8192, vocab_size=1000, rope_theta=1e6, rms_norm_eps=1e-6,
              tie_word_embeddings=False, max_position_embeddings=8192, use_sliding_window=False, hidden_act="silu", torch_dtype="bfloat16")


def _run(native, steps, **config):
    engine = Engine.from_config(dict(CONFIG, **config), seed=3, dtype="bfloat16", kv_cache_tokens=16384, max_seqs=40, max_batch_size=40,
                                max_batch_tokens=8192, max_model_len=4096)
    model = engine.runner.model
    took = []
    if not native:
        model._prenorm_run = None
    elif model._prenorm_run is not None:
        forward = model._prenorm_run.forward
        model._prenorm_run.forward = lambda *a: took.append(1) or forward(*a)
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
    return out, counts, len(took)


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


def test_models_of_another_kind_keep_their_blocks():
    from inferflux_b200.engine.prenorm_run import PrenormRun
    for other in (dict(head_dim=64), dict(intermediate_size=1024), dict(use_sliding_window=True, sliding_window=64, max_window_layers=0)):
        engine = Engine.from_config(dict(CONFIG, **other), seed=3, dtype="bfloat16", kv_cache_tokens=1024, max_seqs=2, max_model_len=512)
        assert PrenormRun.of(engine.runner.model) is None
