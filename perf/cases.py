"""The work that a program has this library do, as cases that can be timed and checked: whole calls through the engine's
public entry points, from the smallest model on a few tokens to prompts of thousands of tokens and models of 16 GB.

A case names a model, a number format and a kind of call:
  generate: a batch of prompts enters the cache in one step, `new` tokens are decoded behind them, and the logits behind the
            last one are read (open, step, the choice of the first tokens, decode, step, close);
  prefill:  prompts enter the cache in one step and the logits of each one's last token are read;
  score:    the same, with the logits of every position (perplexity, ranking of given texts).

Models are the shapes that the benchmark and the tests of this repository run, with seeded random weights. Layer matrices
are N(0, 0.02). The embedding is larger than what the layers add to it, and the head's rows are the embedding's in another
order (the same order where the configuration ties them), so that the next token is a clear choice, as it is for a trained
model most of the time: a greedy run is the same tokens for every correct implementation, and its logits can be compared."""
import math
import random

import numpy as np
import torch

from etalii.dllm_b200 import Engine, SamplingOptions
from etalii.dllm_b200 import architectures  # noqa: F401  (registers the architectures)
from etalii.dllm_b200.config.registry import architecture

DEVICE = "cuda:0"
PAGE = 64  # positions a cache page holds


def _llama(layers, width, heads, kv_heads, dim, ff, vocab, theta, positions, eps=1e-5, tied=True, scaling=None):
    out = {"model_type": "llama", "num_hidden_layers": layers, "hidden_size": width, "num_attention_heads": heads,
           "num_key_value_heads": kv_heads, "head_dim": dim, "intermediate_size": ff, "vocab_size": vocab,
           "rope_theta": theta, "rms_norm_eps": eps, "tie_word_embeddings": tied, "max_position_embeddings": positions,
           "hidden_act": "silu", "bos_token_id": 1, "eos_token_id": 2}
    if scaling:
        out["rope_scaling"] = scaling
    return out


def _tisalorn(width, heads, dim, ff, layers, vocab):
    decay = [1.0 - 2.0 ** -(5 + 4 * i / max(1, heads - 1)) for i in range(heads)]
    groups = heads // 4
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    kinds = [
        {"type": "parallel", "mlp": mlp, "mixer": {
            "left": {"heads": heads, "kv_heads": groups, "dim": dim, "vdim": dim,
                     "rot": {"base": 500000.0, "dims": dim // 2}, "scale": dim ** -0.5},
            "right": {"heads": heads, "dim": dim, "vdim": dim, "decay": decay}}},
        {"type": "delta", "mlp": mlp, "mixer": {"heads": heads, "kv_heads": groups, "dim": dim, "vdim": dim, "conv": 4}},
        {"type": "lightning", "mlp": mlp, "mixer": {"heads": heads, "dim": dim, "vdim": dim, "decay": decay}}]
    return {"architecture": "Tisalorn", "vocab": vocab, "width": width, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
            "max_position": 8192, "layers": [kinds[i % 3] for i in range(layers)]}


# name: (configuration, standard deviation of the embedding: about twice what the layers add up to)
MODELS = {
    "tiny-llama": (_llama(2, 64, 4, 2, 16, 160, 256, 10000.0, 128), 1.0),
    "smollm2-135m": (_llama(30, 576, 9, 3, 64, 1536, 49152, 100000.0, 8192), 1.0),
    "smollm2-1.7b": (_llama(24, 2048, 32, 32, 64, 8192, 49152, 130000.0, 8192), 4.0),
    "llama-3.1-8b": (_llama(32, 4096, 32, 8, 128, 14336, 128256, 500000.0, 8192, tied=False, scaling={
        "rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
        "original_max_position_embeddings": 8192}), 8.0),
    "tisalorn-2k": (_tisalorn(2048, 16, 128, 8192, 4, 49152), 4.0),
}


def _case(name, kind, model, dtype, batch, shortest, longest, new=0, temperature=0.0, min_p=0.0):
    return {"name": name, "kind": kind, "model": model, "dtype": dtype, "batch": batch, "shortest": shortest,
            "longest": longest, "new": new, "temperature": temperature, "min_p": min_p}


def listed():
    return [
        # the smallest call: a toy model on the 32-bit path, a handful of tokens (a first try, a unit test of a user's)
        _case("tiny_fp32_generate_b3", "generate", "tiny-llama", "float32", 3, 5, 17, 8),
        # one person asks a small model a short question: nothing but the latency of a step
        _case("135m_bf16_generate_b1", "generate", "smollm2-135m", "bfloat16", 1, 16, 16, 64),
        # the headline workload: a batch of unequal prompts, then decoding over contexts of up to two thousand
        _case("135m_bf16_generate_b8", "generate", "smollm2-135m", "bfloat16", 8, 128, 2048, 128),
        # a full batch with sampling, as an offline job runs it
        _case("135m_bf16_generate_b64_sampled", "generate", "smollm2-135m", "bfloat16", 64, 128, 2048, 64, 0.8, 0.05),
        # the headline prompt: time to the first token of one long prompt
        _case("135m_bf16_prefill_2048", "prefill", "smollm2-135m", "bfloat16", 1, 2048, 2048),
        # many short texts of any length scored at every position
        _case("135m_bf16_score_b16", "score", "smollm2-135m", "bfloat16", 16, 1, 143),
        # a larger model, unequal long prompts
        _case("1.7b_bf16_generate_b8", "generate", "smollm2-1.7b", "bfloat16", 8, 512, 4096, 32),
        # the largest model: a long prompt, and one person's answer, which is its weights read once a token
        _case("8b_bf16_prefill_2048", "prefill", "llama-3.1-8b", "bfloat16", 1, 2048, 2048),
        _case("8b_bf16_generate_b1", "generate", "llama-3.1-8b", "bfloat16", 1, 100, 100, 32),
        # the 32-bit path: decoding for reproducible answers, and a long prompt
        _case("135m_fp32_generate_b8", "generate", "smollm2-135m", "float32", 8, 50, 700, 32),
        _case("135m_fp32_prefill_2048", "prefill", "smollm2-135m", "float32", 1, 2048, 2048),
        # an architecture with recurrent memories beside attention: the scans of prompts and of single tokens
        _case("tisalorn_bf16_generate_b8", "generate", "tisalorn-2k", "bfloat16", 8, 128, 2048, 64),
    ]


def draw(rng):
    """One more case of the same ranges: models and calls as above, sizes over their logarithm."""
    def size(low, high):
        return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))

    kind, model, dtype, batches, lengths, new = rng.choice([
        ("generate", "tiny-llama", "float32", (1, 4), (1, 48), (4, 16)),
        ("generate", "smollm2-135m", "bfloat16", (1, 64), (1, 2048), (16, 128)),
        ("generate", "smollm2-135m", "bfloat16", (1, 64), (1, 2048), (16, 128)),
        ("prefill", "smollm2-135m", "bfloat16", (1, 16), (16, 2048), None),
        ("score", "smollm2-135m", "bfloat16", (1, 16), (1, 192), None),
        ("generate", "smollm2-1.7b", "bfloat16", (1, 8), (16, 4096), (8, 32)),
        ("prefill", "llama-3.1-8b", "bfloat16", (1, 2), (64, 1024), None),
        ("generate", "llama-3.1-8b", "bfloat16", (1, 4), (8, 256), (8, 24)),
        ("generate", "smollm2-135m", "float32", (1, 16), (1, 384), (8, 32)),
        ("prefill", "smollm2-135m", "float32", (1, 4), (64, 512), None),
        ("generate", "tisalorn-2k", "bfloat16", (1, 8), (16, 2048), (16, 64)),
    ])
    ends = sorted((size(*lengths), size(*lengths)))
    sampled = kind == "generate" and rng.random() < 0.25
    case = _case("", kind, model, dtype, size(*batches), ends[0], ends[1], 0 if new is None else size(*new),
                 0.8 if sampled else 0.0, 0.05 if sampled else 0.0)
    del case["name"]
    return case


def _lengths(case):
    """The prompts' lengths: spread evenly from the shortest to the longest, in no order."""
    n, low, high = case["batch"], case["shortest"], case["longest"]
    out = [high] if n == 1 else [low + (high - low) * i // (n - 1) for i in range(n)]
    random.Random(n * 1000003 + low * 1009 + high).shuffle(out)
    return out


# ---- weights ------------------------------------------------------------------------------------------------------------


def _layout(config):
    """{tensor name: shape} of a model's checkpoint, in a fixed order."""
    shapes = {}
    if config.get("model_type") == "llama":
        w, ff, d = config["hidden_size"], config["intermediate_size"], config["head_dim"]
        q, kv = config["num_attention_heads"] * d, config["num_key_value_heads"] * d
        for i in range(config["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for name, shape in (("self_attn.q_proj", (q, w)), ("self_attn.k_proj", (kv, w)), ("self_attn.v_proj", (kv, w)),
                                ("self_attn.o_proj", (w, q)), ("mlp.gate_proj", (ff, w)), ("mlp.up_proj", (ff, w)),
                                ("mlp.down_proj", (w, ff)), ("input_layernorm", (w,)), ("post_attention_layernorm", (w,))):
                shapes[p + name + ".weight"] = shape
        shapes["model.norm.weight"] = (w,)
        return shapes
    w = config["width"]
    for i, layer in enumerate(config["layers"]):
        m, ff, p = layer["mixer"], layer["mlp"]["ff"], f"l{i}."
        if layer["type"] == "parallel":
            a, r = m["left"], m["right"]
            shapes.update({p + "mix.left.q": (a["heads"] * a["dim"], w), p + "mix.left.k": (a["kv_heads"] * a["dim"], w),
                           p + "mix.left.o": (w, a["heads"] * a["dim"]), p + "mix.left.out": (w,)})
            inner = r["heads"] * r["dim"]
            shapes.update({p + f"mix.right.{k}": (inner, w) for k in "qkvg"})
            shapes.update({p + "mix.right.o": (w, inner), p + "mix.right.out": (w,)})
        elif layer["type"] == "lightning":
            inner = m["heads"] * m["dim"]
            shapes.update({p + f"mix.{k}": (inner, w) for k in "qkvg"})
            shapes.update({p + "mix.o": (w, inner), p + "mix.norm": (inner,)})
        else:
            inner, qk = m["heads"] * m["vdim"], m["kv_heads"] * m["dim"]
            shapes.update({p + "mix.q": (qk, w), p + "mix.k": (qk, w), p + "mix.v": (inner, w), p + "mix.g": (inner, w),
                           p + "mix.b": (m["heads"], w), p + "mix.a": (m["heads"], w), p + "mix.A_log": (m["heads"],),
                           p + "mix.dt_bias": (m["heads"],), p + "mix.norm": (m["vdim"],), p + "mix.o": (w, inner),
                           p + "mix.q.conv": (qk, m["conv"]), p + "mix.k.conv": (qk, m["conv"]),
                           p + "mix.v.conv": (inner, m["conv"])})
        shapes.update({p + "mlp.gate": (ff, w), p + "mlp.up": (ff, w), p + "mlp.down": (w, ff), p + "norm1": (w,),
                       p + "norm2": (w,)})
    shapes["final.norm"] = (w,)
    return shapes


def _sizes(config):
    """(width, vocabulary, whether the head is the embedding)."""
    if config.get("model_type") == "llama":
        return config["hidden_size"], config["vocab_size"], config["tie_word_embeddings"]
    return config["width"], config["vocab"], False


def _successor(config, seed):
    """The token that follows each token where the embedding alone decides: itself with a tied head."""
    _, vocab, tied = _sizes(config)
    return np.arange(vocab) if tied else np.random.default_rng(seed + 77).permutation(vocab)


def _weights(model, seed):
    """A checkpoint's tensors in bfloat16, on the device."""
    config, spread = MODELS[model]
    width, vocab, tied = _sizes(config)
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed(seed * 7919 + 13)

    def normal(shape):
        return torch.randn(shape, generator=generator, device=DEVICE, dtype=torch.bfloat16)

    out = {}
    for name, shape in _layout(config).items():
        if name.endswith("A_log"):  # decays of 1 to 16, step sizes of 0.001 to 0.1, as such models are initialised
            out[name] = torch.log(1 + 15 * torch.rand(shape, generator=generator, device=DEVICE)).bfloat16()
        elif name.endswith("dt_bias"):
            step = torch.exp(torch.rand(shape, generator=generator, device=DEVICE) * math.log(100.0)) * 0.001
            out[name] = (step + torch.log(-torch.expm1(-step))).bfloat16()
        elif name.endswith(".conv"):
            out[name] = normal(shape) * 0.3
        elif len(shape) == 1:
            out[name] = (1.0 + 0.01 * normal(shape).float()).bfloat16()
        else:
            out[name] = normal(shape) * 0.02
    final = "model.norm.weight" if "model.norm.weight" in out else "final.norm"
    # (the chosen token's logit comes to about 20; a tied head's rows are `spread` times as large)
    out[final] = (out[final].float() * (25.0 / width / (spread if tied else 1.0))).bfloat16()
    embed, head = ("model.embed_tokens.weight", "lm_head.weight") if final == "model.norm.weight" else ("embed", "head")
    out[embed] = normal((vocab, width)) * spread
    if not tied:
        rows = torch.empty(vocab, dtype=torch.long)
        rows[torch.from_numpy(_successor(config, seed))] = torch.arange(vocab)
        out[head] = (out[embed].float() / spread)[rows.to(DEVICE)].bfloat16()
    return out


def _prompts(case, seed):
    vocab = _sizes(MODELS[case["model"]][0])[1]
    rng = np.random.default_rng(seed)
    return [rng.integers(0, vocab, n).tolist() for n in _lengths(case)]


# ---- the calls ----------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    config_dict, _ = MODELS[case["model"]]
    name = config_dict.get("model_type") or config_dict["architecture"]
    config = architecture(name).config_class.from_hf(config_dict, None)
    prompts = _prompts(case, seed)
    room = sum(-(-(len(p) + case["new"] + 1) // PAGE) * PAGE for p in prompts)
    engine = Engine(config, _weights(case["model"], seed), dtype=case["dtype"], device=DEVICE, max_tokens=room,
                    max_slots=len(prompts))
    options = SamplingOptions(temperature=case["temperature"], min_p=case["min_p"], seed=seed)
    return {"case": case, "engine": engine, "prompts": prompts, "options": options}


def run(state):
    case, engine, prompts, options = state["case"], state["engine"], state["prompts"], state["options"]
    slots = engine.open(len(prompts))
    if case["kind"] != "generate":
        want = [list(range(len(p))) for p in prompts] if case["kind"] == "score" else None
        logits = engine.step(slots, prompts, want)
        engine.close(slots)
        return {"logits": logits}
    if options.temperature > 0:
        engine.sampler.seed(slots, [options.seed + i for i in range(len(slots))])
    first = engine.step(slots, prompts).clone()  # (a work buffer: the next step overwrites it)
    tokens = engine.sampler.choose(first, engine.last_batch.slots, options).tolist()
    chosen = [tokens] + engine.decode(slots, tokens, case["new"], options)
    logits = engine.step(slots, [[t] for t in chosen[-1]])
    engine.close(slots)
    return {"first": first, "tokens": torch.tensor(chosen, dtype=torch.int32), "logits": logits}


# ---- what a call cannot do without --------------------------------------------------------------------------------------


def work(case):
    """Every weight that a step uses read once a step (no step can begin before the one before it has ended), the keys,
    values and states of the live sequences read once a step, logits written once; products and attention of all tokens."""
    config, _ = MODELS[case["model"]]
    width, vocab, _ = _sizes(config)
    size = 2 if case["dtype"] == "bfloat16" else 4
    lengths, steps = _lengths(case), case["new"] + 1 if case["kind"] == "generate" else 0
    layer_values = sum(math.prod(s) for s in _layout(config).values())
    head_values = width * vocab
    if config.get("model_type") == "llama":
        layers, heads, d = config["num_hidden_layers"], config["num_attention_heads"], config["head_dim"]
        kv_row, pair = 2 * layers * config["num_key_value_heads"] * d * size, 4 * layers * heads * d
        state, state_flops = 0, 0
    else:
        m = [layer["mixer"] for layer in config["layers"]]
        softmax = [x["left"] for x in m if "left" in x]
        memories = [x.get("right", x) for x in m]
        kv_row = sum(2 * a["kv_heads"] * a["dim"] * size for a in softmax)
        pair = sum(4 * a["heads"] * a["dim"] for a in softmax)
        state = 2 * 4 * sum(a["heads"] * a["dim"] * a["vdim"] for a in memories)  # read and written, 32 bits
        state_flops = sum(4 * a["heads"] * a["dim"] * a["vdim"] for a in memories)
    tokens = sum(lengths)
    rows = tokens if case["kind"] == "score" else len(lengths)
    nbytes = (layer_values + head_values) * size + tokens * kv_row + rows * vocab * 4 + len(lengths) * state / 2
    flops = 2 * layer_values * tokens + 2 * head_values * rows + sum(pair * n * (n + 1) / 2 for n in lengths) \
        + state_flops * tokens
    for step in range(steps):
        context = sum(n + step + 1 for n in lengths)
        nbytes += (layer_values + head_values) * size + context * kv_row + len(lengths) * state
        flops += len(lengths) * (2 * (layer_values + head_values) + state_flops) + pair * context
    if steps:
        nbytes += len(lengths) * vocab * 4
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """About four times what a call is off by from `exact` on a B200. The 32-bit path: 7e-7 through 30 layers. bfloat16
    (operands, keys and values are rounded, sums are not): 0.003 at the smallest shape, more for deeper and wider ones."""
    if case["dtype"] == "float32":
        return {"rel": 3e-6, "differ": 0.0}
    return {"rel": {"smollm2-1.7b": 0.017, "llama-3.1-8b": 0.028}.get(case["model"], 0.012), "differ": 0.005}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, weight, eps):
    return _rms(x - x.mean(-1, keepdim=True), eps) * weight


def _causal(q, k, v, scale):
    """q [n, heads, d], k and v [n, kv heads, d]: causal softmax attention, a kv head at a time."""
    n, heads, d = q.shape
    group = heads // k.shape[1]
    unseen = torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1)
    out = torch.empty_like(q)
    for g in range(k.shape[1]):
        mine = slice(g * group, (g + 1) * group)
        scores = torch.einsum("thd,sd->hts", q[:, mine], k[:, g]) * scale
        weights = torch.softmax(scores.masked_fill_(unseen, -math.inf), -1)
        out[:, mine] = torch.einsum("hts,sd->thd", weights, v[:, g])
    return out.reshape(n, heads * d)


def _llama_hidden(config, w, x):
    d, heads, groups = config["head_dim"], config["num_attention_heads"], config["num_key_value_heads"]
    eps, scaling = config["rms_norm_eps"], config.get("rope_scaling")
    frequency = config["rope_theta"] ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    if scaling:
        wavelength, whole = 2 * math.pi / frequency, scaling["original_max_position_embeddings"]
        low, high = scaling["low_freq_factor"], scaling["high_freq_factor"]
        part = ((whole / wavelength - low) / (high - low)).clamp(0, 1)
        frequency = (1 - part) * frequency / scaling["factor"] + part * frequency
    angle = torch.arange(len(x), dtype=torch.float64, device=x.device)[:, None, None] * frequency
    cos, sin = angle.cos(), angle.sin()

    def turn(y):
        a, b = y[..., :d // 2], y[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for i in range(config["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w(p + "input_layernorm.weight")
        q = turn((h @ w(p + "self_attn.q_proj.weight").T).view(-1, heads, d))
        k = turn((h @ w(p + "self_attn.k_proj.weight").T).view(-1, groups, d))
        v = (h @ w(p + "self_attn.v_proj.weight").T).view(-1, groups, d)
        x = x + _causal(q, k, v, d ** -0.5) @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
        gate = h @ w(p + "mlp.gate_proj.weight").T
        x = x + (torch.nn.functional.silu(gate) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    return _rms(x, eps) * w("model.norm.weight")


def _decayed(q, k, v, decay):
    """S <- decay S + k v^T, o = S^T q per head, written out over all earlier positions."""
    n, heads, _ = q.shape
    age = torch.arange(n, dtype=torch.float64, device=q.device)
    age = age[:, None] - age[None, :]
    out = torch.empty_like(v)
    for h in range(heads):
        share = torch.where(age >= 0, torch.exp(age.clamp(min=0) * math.log(decay[h])), 0.0)
        out[:, h] = ((q[:, h] @ k[:, h].T) * share) @ v[:, h]
    return out


def _convolved(x, taps):
    """Causal filter per channel over time, the last tap on the current token; silu behind it."""
    width = taps.shape[1]
    line = torch.cat([x.new_zeros(width - 1, x.shape[1]), x])
    return torch.nn.functional.silu(sum(line[j:j + len(x)] * taps[:, j] for j in range(width)))


def _delta(w, p, m, h, eps):
    n, heads, groups, d, vd = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    share = heads // groups

    def unit(y):
        return y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)

    q, k, v = (_convolved(h @ w(p + name).T, w(p + name + ".conv")) for name in "qkv")
    q = (unit(q.view(n, groups, d)) * d ** -0.5).repeat_interleave(share, 1)
    k = unit(k.view(n, groups, d)).repeat_interleave(share, 1)
    v = v.view(n, heads, vd)
    beta = torch.sigmoid(h @ w(p + "b").T)[..., None]
    keep = torch.exp(-torch.exp(w(p + "A_log")) * torch.nn.functional.softplus(h @ w(p + "a").T + w(p + "dt_bias")))
    keep = keep[..., None, None]
    state, out = h.new_zeros(heads, d, vd), torch.empty_like(v)
    for t in range(n):
        state = state * keep[t]
        u = beta[t] * (v[t] - torch.bmm(k[t, :, None], state)[:, 0])
        state.baddbmm_(k[t][:, :, None], u[:, None])
        out[t] = torch.bmm(q[t, :, None], state)[:, 0]
    out = (_rms(out, eps) * w(p + "norm")).reshape(n, heads * vd)
    return (out * torch.nn.functional.silu(h @ w(p + "g").T)) @ w(p + "o").T


def _tisalorn_mixer(w, p, layer, h, eps):
    m, n, silu = layer["mixer"], len(h), torch.nn.functional.silu
    if layer["type"] == "delta":
        return _delta(w, p, m, h, eps)
    if layer["type"] == "lightning":
        q, k, v = (silu(h @ w(p + name).T).view(n, m["heads"], -1) for name in "qkv")
        o = _rms(_decayed(q, k, v, m["decay"]).reshape(n, -1), eps) * w(p + "norm")
        return (o * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T
    a, r = m["left"], m["right"]
    rot = a["rot"]["dims"]
    frequency = a["rot"]["base"] ** (-torch.arange(0, rot, 2, dtype=torch.float64, device=h.device) / rot)
    angle = torch.arange(n, dtype=torch.float64, device=h.device)[:, None, None] * frequency
    cos, sin = angle.cos(), angle.sin()

    def turn(y):  # neighbouring dimensions are a pair; those behind the rotated ones stay
        even, odd = y[..., 0:rot:2], y[..., 1:rot:2]
        pairs = torch.stack([even * cos - odd * sin, odd * cos + even * sin], -1)
        return torch.cat([pairs.flatten(-2), y[..., rot:]], -1)

    q = (h @ w(p + "left.q").T).view(n, a["heads"], a["dim"])
    k = (h @ w(p + "left.k").T).view(n, a["kv_heads"], a["dim"])
    left = _causal(turn(q), turn(k), k, a["scale"]) @ w(p + "left.o").T
    q, k, v = ((h @ w(p + "right." + name).T).view(n, r["heads"], -1) for name in "qkv")
    o = _rms(_decayed(q, k * r["dim"] ** -0.5, v, r["decay"]), eps).reshape(n, -1)
    right = (o * silu(h @ w(p + "right.g").T)) @ w(p + "right.o").T
    return 0.5 * (_rms(left, eps) * w(p + "left.out") + _rms(right, eps) * w(p + "right.out"))


def _tisalorn_hidden(config, w, x):
    eps = config["norm"]["eps"]
    for i, layer in enumerate(config["layers"]):
        p, limit = f"l{i}.", layer["mlp"]["limit"]
        x = x + _tisalorn_mixer(w, p + "mix.", layer, _layer_norm(x, w(p + "norm1"), eps), eps)
        h = _layer_norm(x, w(p + "norm2"), eps)
        g = (h @ w(p + "mlp.gate").T).clamp(max=limit)
        u = (h @ w(p + "mlp.up").T).clamp(-limit, limit)
        x = x + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(p + "mlp.down").T
    return _layer_norm(x, w("final.norm"), eps)


def exact(case, seed):
    """Whole sequences in float64. What a generating run chooses is the sequence whose every token is the largest logit
    behind the one before it: the successor of each token is put down first, and put right until that holds."""
    config, _ = MODELS[case["model"]]
    tensors, prompts = _weights(case["model"], seed), _prompts(case, seed)
    llama = config.get("model_type") == "llama"
    hidden_of = _llama_hidden if llama else _tisalorn_hidden
    embed = tensors["model.embed_tokens.weight" if llama else "embed"]
    head = embed if _sizes(config)[2] else tensors["lm_head.weight" if llama else "head"]
    head = head.double()
    successor = _successor(config, seed)
    kept = {}
    small = sum(t.numel() for t in tensors.values()) < 3e9  # (a copy in 64 bits is kept where it fits easily)

    def w(name):
        if name in kept:
            return kept[name]
        value = tensors[name].double()
        if small:
            kept[name] = value
        return value

    def logits_of(tokens, rows):
        x = embed[torch.tensor(tokens, device=DEVICE)].double()
        return hidden_of(config, w, x)[rows] @ head.T

    if case["kind"] != "generate":
        rows = slice(None) if case["kind"] == "score" else slice(-1, None)
        return {"logits": torch.cat([logits_of(p, rows) for p in prompts])}
    firsts, lasts, chosen = [], [], []
    for prompt in prompts:
        behind = [prompt[-1]]
        while len(behind) < case["new"] + 2:
            behind.append(int(successor[behind[-1]]))
        behind = behind[1:]
        for _ in range(len(behind) + 1):
            logits = logits_of(prompt + behind, slice(len(prompt) - 1, None))
            best = logits.argmax(-1).tolist()
            wrong = next((i for i, token in enumerate(behind) if best[i] != token), None)
            if wrong is None:
                break
            behind = behind[:wrong] + [best[wrong]]
            while len(behind) < case["new"] + 1:
                behind.append(int(successor[behind[-1]]))
        firsts.append(logits[0])
        lasts.append(logits[-1])
        chosen.append(behind)
    return {"first": torch.stack(firsts), "tokens": torch.tensor(chosen, dtype=torch.int32).T.contiguous(),
            "logits": torch.stack(lasts)}
