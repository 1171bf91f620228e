"""The work this engine is measured by: what serving programs have it do, through its public entry points.

Every case is one of six kinds of work:

* ``decode``: one step of single tokens for requests that are all in the cache, the step a serving loop spends its
  life in.  A pass moves every request one token on, like the real thing; a request that has used up its room starts
  over from its prompt.
* ``prefill``: new prompts, whole or in portions of ``portion`` tokens, to the logits behind their last tokens; the
  requests end with the pass.
* ``mixed``: a scheduler's step while requests come and go: one portion of a new prompt beside decoding requests.
* ``sample``: the next tokens of a step's logits, requests with and without top-k, top-p, min-p, some greedy.

The models are the sizes that the benchmark knows (Qwen2.5 3B, 7B and 14B layer shapes, and the Zetivik design at the
same widths), with random weights; ``layers`` is how many of a size's layers are there.  Layers are all alike; six of
them keep what 16-bit roundings do to the logits of random weights near one part in a hundred (with all 28 of the 7B
size it is four), so that two correct ways of computing a step can be told from a wrong one.
"""
import math

import numpy as np
import torch

from inferflux_b200 import Engine, EngineConfig, SamplingParams, StepEntry, load_config
from inferflux_b200.config import build_spec
from inferflux_b200.engine.model import Model
from inferflux_b200.sampling import Sampler

DEVICE = "cuda:0"
HEAD = 128                  # the size of a head everywhere
ROOM = 2048                 # tokens that a decoding request may grow by before it starts over
#: layers, width, heads, kv heads, feed-forward width, vocabulary, tied output head
SIZES = {
    "3b": (36, 2048, 16, 2, 11008, 151936, True),
    "7b": (28, 3584, 28, 4, 18944, 152064, False),
    "14b": (48, 5120, 40, 8, 13824, 152064, False),
}


def listed():
    q = dict(model="qwen2", dtype="bfloat16")
    z = dict(model="zetivik", dtype="bfloat16")
    return [
        # one person in a conversation: the wait for each token
        dict(q, name="decode_1", kind="decode", size="7b", layers=6, batch=1, shortest=4096, longest=4096),
        # the benchmark's headline step
        dict(q, name="decode_8", kind="decode", size="7b", layers=6, batch=8, shortest=4096, longest=4096),
        # a server under load: many requests, contexts of every length
        dict(q, name="decode_64", kind="decode", size="7b", layers=6, batch=64, shortest=500, longest=3600),
        # a smaller model, an odd number of requests
        dict(q, name="decode_23_small", kind="decode", size="3b", layers=8, batch=23, shortest=90, longest=2100),
        # the benchmark's prompt
        dict(q, name="prefill_2048", kind="prefill", size="7b", layers=6, batch=1, prompt=2048, portion=2048),
        # a short question to a small model: time to the first token
        dict(q, name="prompt_77", kind="prefill", size="3b", layers=8, batch=1, prompt=77, portion=2048),
        # a long document, in portions
        dict(q, name="document_16385", kind="prefill", size="7b", layers=6, batch=1, prompt=16385, portion=2048),
        # a portion of a new prompt beside decoding requests
        dict(q, name="mixed_509_31", kind="mixed", size="7b", layers=6, batch=31, shortest=130, longest=2000, portion=509),
        # the 32-bit path: reference logits for a short prompt
        dict(q, name="float32_301", kind="prefill", size="3b", layers=4, batch=1, prompt=301, portion=2048, dtype="float32"),
        # sampled tokens for a full batch
        dict(name="sample_64", kind="sample", size="7b", rows=64),
        # a design whose layers keep states: a prompt, and the headline step
        dict(z, name="states_prefill_2048", kind="prefill", size="7b", layers=8, batch=1, prompt=2048, portion=2048),
        dict(z, name="states_decode_8", kind="decode", size="7b", layers=8, batch=8, shortest=4096, longest=4096),
    ]


def _log_int(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    """A case of the ranges above: every kind and model, odd sizes, fewer layers where the sizes are large."""
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "prefill", "mixed", "sample"])
    size = rng.choice(["3b", "7b", "7b", "14b"])
    if kind == "sample":
        return dict(kind=kind, size=size, rows=_log_int(rng, 1, 64))
    model = rng.choice(["qwen2", "qwen2", "qwen2", "zetivik"])
    case = dict(kind=kind, model=model, dtype="bfloat16", size=size, layers=rng.randint(3, 7))
    if kind == "prefill" and model == "qwen2" and rng.random() < 0.25:
        return dict(case, size="3b", layers=rng.randint(2, 4), dtype="float32", batch=1, prompt=_log_int(rng, 16, 400), portion=2048)
    if kind == "prefill":
        prompt = _log_int(rng, 20, 8000 if model == "qwen2" else 3000)
        return dict(case, batch=rng.randint(1, 3) if prompt < 1500 else 1, prompt=prompt, portion=rng.choice([512, 1024, 2048]))
    longest = _log_int(rng, 64, 4096)
    case.update(batch=_log_int(rng, 1, 64 if model == "qwen2" else 16), shortest=max(16, longest // rng.choice([1, 2, 8])), longest=longest)
    if kind == "mixed":
        case["portion"] = _log_int(rng, 16, 1024)
    return case


# ------------------------------------------------------------------ models
def _config(case):
    _, hidden, heads, kv_heads, inter, vocab, tied = SIZES[case["size"]]
    if case["model"] == "qwen2":
        return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", hidden_size=hidden, num_hidden_layers=case["layers"],
                    num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=HEAD, intermediate_size=inter,
                    vocab_size=vocab, rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=tied,
                    max_position_embeddings=32768, use_sliding_window=False, hidden_act="silu", torch_dtype="bfloat16")
    ff = dict(kind="dense", ff=inter, limit=7.0)
    left = dict(heads=heads, kv_heads=kv_heads, dim=HEAD, vdim=HEAD, scale=HEAD ** -0.5, mask=dict(size=8192), rot=dict(dims=HEAD, base=500000.0))
    right = dict(heads=heads // 2, kv_heads=heads // 4, dim=HEAD, vdim=HEAD, conv=4)
    pair = dict(type="parallel", mixer=dict(left=left, right=right, left_scale=1.0, right_scale=1.0), mlp=ff)
    lightning = dict(type="lightning", mlp=ff, mixer=dict(heads=heads, dim=HEAD, vdim=HEAD,
                                                          decay=[1.0 - 0.2 * 0.5 ** (8.0 * i / heads) for i in range(heads)]))
    return dict(architecture="Zetivik", width=hidden, vocab=vocab, norm=dict(eps=1e-6), logit_softcap=30.0,
                layers=[pair if i % 2 == 0 else lightning for i in range(case["layers"])])


def _shapes(case):
    """name -> (shape, mean, standard deviation) of every tensor of the model."""
    _, hidden, heads, kv_heads, inter, vocab, tied = SIZES[case["size"]]
    nq, nkv = heads * HEAD, kv_heads * HEAD
    out = {}

    def mat(name, *shape, mean=0.0, std=0.02):
        out[name] = (shape, mean, std)

    if case["model"] == "qwen2":
        mat("model.embed_tokens.weight", vocab, hidden)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            for leaf, rows in (("q", nq), ("k", nkv), ("v", nkv)):
                mat(f"{p}self_attn.{leaf}_proj.weight", rows, hidden)
                mat(f"{p}self_attn.{leaf}_proj.bias", rows)
            mat(p + "self_attn.o_proj.weight", hidden, nq)
            mat(p + "mlp.gate_proj.weight", inter, hidden)
            mat(p + "mlp.up_proj.weight", inter, hidden)
            mat(p + "mlp.down_proj.weight", hidden, inter)
            mat(p + "input_layernorm.weight", hidden, mean=1.0)
            mat(p + "post_attention_layernorm.weight", hidden, mean=1.0)
        mat("model.norm.weight", hidden, mean=1.0)
        if not tied:
            mat("lm_head.weight", vocab, hidden)
        return out
    mat("embed", vocab, hidden)
    for i in range(case["layers"]):
        m = f"l{i}.mix."
        if i % 2 == 0:
            for leaf, rows in (("q", nq), ("k", nkv), ("v", nkv)):
                mat(f"{m}left.{leaf}", rows, hidden)
                mat(f"{m}left.{leaf}.b", rows)
            mat(m + "left.q.norm", HEAD, mean=1.0)
            mat(m + "left.k.norm", HEAD, mean=1.0)
            mat(m + "left.g", heads, hidden)
            mat(m + "left.o", hidden, nq)
            rh, rk = heads // 2, heads // 4
            for leaf, rows in (("q", rk), ("k", rk), ("v", rh)):
                mat(f"{m}right.{leaf}", rows * HEAD, hidden)
                mat(f"{m}right.{leaf}.conv", rows * HEAD, 4, std=0.5)
            mat(m + "right.a", rh, hidden)
            mat(m + "right.b", rh, hidden)
            mat(m + "right.A_log", rh, std=0.5)
            mat(m + "right.dt_bias", rh, std=0.5)
            mat(m + "right.g", rh * HEAD, hidden)
            mat(m + "right.norm", HEAD, mean=1.0)
            mat(m + "right.o", hidden, rh * HEAD)
        else:
            for leaf in "qkvg":
                mat(m + leaf, nq, hidden)
            mat(m + "norm", nq, mean=1.0)
            mat(m + "o", hidden, nq)
        mat(f"l{i}.norm1", hidden, std=0.1)
        mat(f"l{i}.norm2", hidden, std=0.1)
        mat(f"l{i}.mlp.gate", inter, hidden)
        mat(f"l{i}.mlp.up", inter, hidden)
        mat(f"l{i}.mlp.down", hidden, inter)
    mat("final.norm", hidden, std=0.1)
    return out


def _weights(case, seed, only=None):
    """The model's tensors, stored in 16 bits as a checkpoint's are (widened for the 32-bit path).  Each has a seed
    of its own, so that a few of them can be had alone (``only``: the names that begin so)."""
    wide = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    out = {}
    for k, (name, (shape, mean, std)) in enumerate(_shapes(case).items()):
        if only is not None and not name.startswith(only):
            continue
        gen = torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + k) & 0x7FFFFFFFFFFF)
        t = torch.randn(shape, generator=gen, dtype=torch.bfloat16, device=DEVICE).mul_(std)
        if mean:
            t += mean
        out[name] = t.to(wide)
    return out


def _lengths(case):
    """The decoding requests' lengths, spread from the shortest to the longest and not in order."""
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    spread = [hi if n == 1 else lo + (hi - lo) * i // (n - 1) for i in range(n)]
    return [spread[(i * 7) % n] if n % 7 else spread[i] for i in range(n)]


def _tokens(case, seed, index, count):
    vocab = SIZES[case["size"]][5]
    return np.random.RandomState((seed * 4099 + index) % (1 << 32)).randint(0, vocab, count).tolist()


# ------------------------------------------------------------------ a user's program
def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    config = load_config(_config(case))
    model = Model(build_spec(config), torch.float32 if case["dtype"] == "float32" else torch.bfloat16, DEVICE)
    model.load(_weights(case, seed))
    state = dict(case=case, seed=seed)
    page = 16
    pages = lambda n: (n + page - 1) // page
    need = 0
    if case["kind"] != "prefill":
        state["prompts"] = [_tokens(case, seed, i, n) for i, n in enumerate(_lengths(case))]
        state["next"] = [_tokens(case, seed, 1000 + i, ROOM) for i in range(case["batch"])]
        state["rids"] = [f"r{i}" for i in range(case["batch"])]
        need += sum(pages(len(p) + ROOM) for p in state["prompts"])
    if case["kind"] == "prefill":
        state["new"] = [_tokens(case, seed, 2000 + i, case["prompt"]) for i in range(case["batch"])]
        need += case["batch"] * pages(case["prompt"])
    elif case["kind"] == "mixed":
        state["new"] = [_tokens(case, seed, 2000, case["portion"])]
        need += pages(case["portion"])
    state["engine"] = Engine(model, config, EngineConfig(
        dtype=case["dtype"], device=DEVICE, kv_cache_tokens=(need + 1) * page, max_seqs=case["batch"] + 2,
        max_batch_size=case["batch"] + 2, max_model_len=32768))
    if case["kind"] != "prefill":
        _fill(state)
    return state


def _fill(state):
    """The decoding requests' prompts go into the cache, several to a step."""
    engine = state["engine"]
    batch, size = [], 0
    for rid, prompt in zip(state["rids"], state["prompts"]):
        for at in range(0, len(prompt), 2048):
            part = prompt[at:at + 2048]
            if batch and (size + len(part) > 8192 or batch[-1].rid == rid):
                engine.run_step(batch)
                batch, size = [], 0
            batch.append(StepEntry(rid, part, []))
            size += len(part)
    engine.run_step(batch)
    state["turn"] = 0


def _prepare_sample(case, seed):
    vocab, rows = SIZES[case["size"]][5], case["rows"]
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kinds = [dict(temperature=0.8, top_p=0.95), dict(temperature=1.0), dict(temperature=0.7, top_k=40, top_p=0.9),
             dict(temperature=0.0), dict(temperature=0.9, min_p=0.05), dict(temperature=1.0, top_k=100)]
    return dict(case=case, logits=torch.randn((rows, vocab), generator=gen, device=DEVICE) * 2.5, sampler=Sampler(vocab, DEVICE),
                params=[SamplingParams(**kinds[i % len(kinds)]) for i in range(rows)],
                seeds=[seed * 77 + i for i in range(rows)], counters=[3 * i for i in range(rows)], recent=[[]] * rows)


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return state["sampler"].sample(state["logits"], state["params"], state["seeds"], state["counters"], state["recent"])
    engine = state["engine"]
    if case["kind"] == "prefill":
        at, step, end = 0, case["portion"], case["prompt"]
        while at < end:
            n = min(step, end - at)
            want = [n - 1] if at + n == end else []
            logits = engine.run_step([StepEntry(f"new{i}", p[at:at + n], want) for i, p in enumerate(state["new"])])
            at += n
        for i in range(len(state["new"])):
            engine.end_request(f"new{i}")
        return _answer(logits)
    if state["turn"] == ROOM:
        for rid in state["rids"]:
            engine.end_request(rid)
        _fill(state)
    turn = state["turn"]
    state["turn"] = turn + 1
    entries = [StepEntry(rid, [nxt[turn]], [0]) for rid, nxt in zip(state["rids"], state["next"])]
    if case["kind"] == "mixed":
        entries.append(StepEntry("new", state["new"][0], [case["portion"] - 1]))
    logits = engine.run_step(entries)
    if case["kind"] == "mixed":
        engine.end_request("new")
    return _answer(logits)


def _answer(logits):
    """The logits: the first request's, and the others'."""
    return {"first": logits[:1], "others": logits[1:]} if logits.shape[0] > 1 else {"first": logits}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    _, hidden, heads, kv_heads, inter, vocab, _ = SIZES[case["size"]]
    if case["kind"] == "sample":
        return {"bytes": 4 * case["rows"] * vocab + 4 * case["rows"], "flops": 0}
    elt = 4 if case["dtype"] == "float32" else 2
    sizes = {name: math.prod(shape) for name, (shape, _, _) in _shapes(case).items()}
    embed = "model.embed_tokens.weight" if case["model"] == "qwen2" else "embed"
    head = "lm_head.weight" if "lm_head.weight" in sizes else embed
    body = sum(n for name, n in sizes.items() if name not in (embed, head))
    attending = case["layers"] if case["model"] == "qwen2" else (case["layers"] + 1) // 2
    cached = 2 * kv_heads * HEAD * elt * attending                       # bytes of a token's keys and values
    pair = 4 * heads * HEAD * attending                                  # operations of one query and one key
    state_bytes = state_flops = 0                                        # a request's states, and what a token does to them
    if case["model"] == "zetivik":
        cells = (heads // 2 * attending + heads * (case["layers"] - attending)) * HEAD * HEAD
        state_bytes, state_flops = 2 * 4 * cells, 6 * cells
    new, bytes_, flops, rows = 0, 0, 0, 0
    if case["kind"] != "prefill":
        lengths = _lengths(case)
        new += len(lengths)
        rows += len(lengths)
        bytes_ += sum(lengths) * cached + len(lengths) * state_bytes
        flops += sum(n + 1 for n in lengths) * pair
    if case["kind"] != "decode":
        n, count = (case["prompt"], case["batch"]) if case["kind"] == "prefill" else (case["portion"], 1)
        new += n * count
        rows += count
        bytes_ += count * (n * cached + state_bytes)                     # written once; read back from on-chip memory at best
        flops += count * n * (n + 1) // 2 * pair
    bytes_ += elt * (body + sizes[head] + new * hidden) + new * cached + 4 * rows * vocab
    flops += 2 * body * new + 2 * sizes[head] * rows + state_flops * new
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4}          # 4.8e-6 off the result in 64 bits
    # One to two parts in a hundred off the result in 64 bits (rms); two such results differ by up to the root of
    # two more, and the largest of 152,064 differences is five times their rms.
    return {"rel": 3e-2, "max": 0.3}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    """The first request's logits in 64 bits (the others' would only take longer)."""
    if case["kind"] == "sample":
        return None
    if case["kind"] == "prefill":
        tokens, alone = _tokens(case, seed, 2000, case["prompt"]), case["batch"] == 1
    else:
        tokens = _tokens(case, seed, 0, _lengths(case)[0]) + _tokens(case, seed, 1000, ROOM)[:1]
        alone = case["kind"] == "decode" and case["batch"] == 1
    forward = _qwen2_logits if case["model"] == "qwen2" else _zetivik_logits
    logits = forward(case, seed, torch.tensor(tokens, device=DEVICE))
    return {"first": logits} if alone else {"first": logits, "others": None}


def _rms(v, eps=1e-6):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def _rotated(x, positions, base):
    """x [T, heads, HEAD]: dimensions (i, i + HEAD/2) turn by position * base^(-2i/HEAD)."""
    half = HEAD // 2
    f = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / HEAD)
    a = (positions.double()[:, None] * f)[:, None, :]
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1)


def _attention(q, k, v, chunk=None):
    """Causal attention of the last rows: q [Tq, heads, HEAD], k and v [T, kv heads, HEAD] (inside stretches of ``chunk``)."""
    tq, t, group = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    pos, out = torch.arange(t, device=q.device), torch.empty_like(q)
    for at in range(0, tq, 1024):
        rows = pos[t - tq + at:t - tq + min(tq, at + 1024)]
        hidden = rows[:, None] < pos[None, :]
        if chunk:
            hidden |= (rows[:, None] // chunk) != (pos[None, :] // chunk)
        for kv in range(k.shape[1]):
            s = torch.einsum("qhd,kd->hqk", q[at:at + 1024, kv * group:(kv + 1) * group], k[:, kv]) * HEAD ** -0.5
            p = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1)
            out[at:at + 1024, kv * group:(kv + 1) * group] = torch.einsum("hqk,kd->qhd", p, v[:, kv])
    return out


def _doubles(case, seed, prefix):
    """The tensors whose names begin so, by the rest of their names, in 64 bits."""
    return {name[len(prefix):]: t.double() for name, t in _weights(case, seed, prefix).items()}


def _row_blocks(fn, x):
    """fn over a few thousand rows at a time (what lies between is large in 64 bits)."""
    return torch.cat([fn(part) for part in x.split(4096)])


def _qwen2_logits(case, seed, tokens):
    pos = torch.arange(len(tokens), device=DEVICE)
    x = _weights(case, seed, "model.embed_tokens")["model.embed_tokens.weight"][tokens].double()
    for i in range(case["layers"]):
        w = _doubles(case, seed, f"model.layers.{i}.")
        h = _rms(x) * w["input_layernorm.weight"]
        if i == case["layers"] - 1:                    # only the last token's result is wanted
            x, last = x[-1:], 1
        else:
            last = len(tokens)
        proj = lambda rows, leaf: (rows @ w[f"self_attn.{leaf}_proj.weight"].T + w[f"self_attn.{leaf}_proj.bias"]).reshape(rows.shape[0], -1, HEAD)
        q = _rotated(proj(h[-last:], "q"), pos[-last:], 1e6)
        o = _attention(q, _rotated(proj(h, "k"), pos, 1e6), proj(h, "v"))
        x = x + o.reshape(last, -1) @ w["self_attn.o_proj.weight"].T
        h = _rms(x) * w["post_attention_layernorm.weight"]
        glu = lambda rows: (torch.nn.functional.silu(rows @ w["mlp.gate_proj.weight"].T) * (rows @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T
        x = x + _row_blocks(glu, h)
    x = _rms(x[-1:]) * _doubles(case, seed, "model.norm.")["weight"]
    head = "model.embed_tokens.weight" if SIZES[case["size"]][6] else "lm_head.weight"
    return x @ _weights(case, seed, head)[head].double().T


def _zetivik_logits(case, seed, tokens):
    heads = SIZES[case["size"]][2]
    t, pos = len(tokens), torch.arange(len(tokens), device=DEVICE)
    embed = _weights(case, seed, "embed")["embed"]
    x = embed[tokens].double()
    silu = torch.nn.functional.silu
    for i in range(case["layers"]):
        w = _doubles(case, seed, f"l{i}.")
        h = _rms(x) * (1.0 + w["norm1"])
        if i % 2 == 0:
            proj = lambda leaf: (h @ w["mix.left." + leaf].T + w[f"mix.left.{leaf}.b"]).reshape(t, -1, HEAD)
            q = _rotated(_rms(proj("q")) * w["mix.left.q.norm"], pos, 500000.0)
            k = _rotated(_rms(proj("k")) * w["mix.left.k.norm"], pos, 500000.0)
            o = _attention(q, k, proj("v"), 8192) * torch.sigmoid(h @ w["mix.left.g"].T)[:, :, None]
            x = x + o.reshape(t, -1) @ w["mix.left.o"].T + _gated_delta(h, w, heads // 2) @ w["mix.right.o"].T
        else:
            q, k, v = (silu(h @ w["mix." + leaf].T).reshape(t, heads, HEAD) for leaf in "qkv")
            o = torch.empty_like(v)
            back = (pos[:, None] - pos[None, :]).double()
            for n in range(heads):
                fade = torch.exp(back * math.log(1.0 - 0.2 * 0.5 ** (8.0 * n / heads))).masked_fill_(back < 0, 0.0)
                o[:, n] = ((q[:, n] @ k[:, n].T) * fade) @ v[:, n]
            o = _rms(o.reshape(t, -1)) * w["mix.norm"] * torch.sigmoid(h @ w["mix.g"].T)
            x = x + o @ w["mix.o"].T
        h = _rms(x) * (1.0 + w["norm2"])
        if i == case["layers"] - 1:
            x, h = x[-1:], h[-1:]

        def glu(rows):
            g, u = (rows @ w["mlp.gate"].T).clamp(max=7.0), (rows @ w["mlp.up"].T).clamp(-7.0, 7.0)
            return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w["mlp.down"].T
        x = x + _row_blocks(glu, h)
    x = _rms(x) * (1.0 + _doubles(case, seed, "final.")["norm"])
    return 30.0 * torch.tanh(x @ embed.double().T / 30.0)


def _gated_delta(h, w, heads):
    """Per head S <- g S, u = beta (v - S^T k), S <- S + k u^T, o = S^T q, token by token, normed and gated."""
    t = h.shape[0]
    rows = {}
    for leaf in "qkv":
        u, taps = h @ w["mix.right." + leaf].T, w[f"mix.right.{leaf}.conv"]
        padded = torch.cat([u.new_zeros((3, u.shape[1])), u])
        y = sum(padded[j:j + t] * taps[:, j] for j in range(4))
        rows[leaf] = torch.nn.functional.silu(y).reshape(t, -1, HEAD)
    unit = lambda v: v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6)
    share = heads // rows["q"].shape[1]
    q = (unit(rows["q"]) * HEAD ** -0.5).repeat_interleave(share, dim=1)
    k = unit(rows["k"]).repeat_interleave(share, dim=1)
    a = torch.nn.functional.softplus(h @ w["mix.right.a"].T + w["mix.right.dt_bias"], threshold=1e4)
    g, beta = torch.exp(-torch.exp(w["mix.right.A_log"]) * a), torch.sigmoid(h @ w["mix.right.b"].T)
    g, v = g[:, :, None, None], rows["v"]
    s, o = h.new_zeros((heads, HEAD, HEAD)), torch.empty_like(v)
    for i in range(t):
        s *= g[i]
        u = beta[i][:, None] * (v[i] - torch.bmm(k[i][:, None, :], s)[:, 0])
        s.baddbmm_(k[i][:, :, None], u[:, None, :])
        o[i] = torch.bmm(q[i][:, None, :], s)[:, 0]
    return (_rms(o) * w["mix.right.norm"]).reshape(t, -1) * torch.nn.functional.silu(h @ w["mix.right.g"].T)
