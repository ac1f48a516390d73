"""The work whose speed this framework is held to: what its users have it do, through the entry points they call.

Two kinds of pass, over models with the layer sizes of this repository's benchmark and random bfloat16 weights:

  session   requests through `NativeStepRunner`: their prompts, packed several to a step (long ones in portions), then decode
            steps of all of them together, with the next token's logits of every request after every step; then the
            requests end.  The tokens are given (a replay), so every step's logits can be compared.
  serve     a list of prompts through `NativeEngine.generate`, greedily: admission, portions of prompts beside decoding
            requests, sampling, tokens back.

A pass starts without any request in the cache and leaves none behind.  The model is loaded once for a process, as a
program that serves it does; a state is a set of prompts.
"""
import functools
import json
import math
import os
import shutil
import struct
import tempfile
from pathlib import Path

import numpy as np
import torch

# ---- models ---------------------------------------------------------------------------------------------------------
QWEN_05B = {
    "architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2",
    "num_hidden_layers": 24, "hidden_size": 896, "num_attention_heads": 14, "num_key_value_heads": 2,
    "intermediate_size": 4864, "vocab_size": 151936, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6,
    "tie_word_embeddings": True, "max_position_embeddings": 32768, "bos_token_id": -1, "eos_token_id": -1,
    "use_sliding_window": False,
}
QWEN_15B = dict(QWEN_05B, num_hidden_layers=28, hidden_size=1536, num_attention_heads=12, intermediate_size=8960)


def _lasizen():
    attention = {"type": "attention", "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                                                "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}}
    delta = {"type": "delta", "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}}
    mlp = {"kind": "dense", "ff": 8192}
    return {"architecture": "Lasizen", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "embedding": {"scale": 2048.0 ** 0.5},
            "logit_scale": 1.0 / 2048.0 ** 0.5, "loop": {"start": 1, "stop": 3, "times": 2},
            "layers": [dict(attention, mlp=mlp), dict(attention, mlp=mlp), dict(delta, mlp=mlp), dict(attention, mlp=mlp)]}


def _zodosun():
    delta = {"type": "general_delta", "mixer": {"heads": 32, "dim": 64, "rank": 64}}
    pair = {"type": "parallel", "mixer": {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "bias_max": 1024,
                                                   "q_temp": {"coef": 0.1, "every": 1024}},
                                          "right": {"heads": 8, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-2 - h) for h in range(8)]}}}
    mlp = {"kind": "dense", "ff": 5504}
    return {"architecture": "Zodosun", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6, "groups": 4}, "logit_scale": 0.5,
            "layers": [dict(m, mlp=mlp) for m in (delta, pair, delta, delta, pair, delta)]}


# The Qwen2 decoder is what the framework is for first; two of the further architectures stand for the other kinds of layers:
# windows and sinks, gated delta rules, token shifts; delta rules with a decay per channel, sigmoid weights, linear attention.
# (Routed experts are left out: two correct implementations choose another expert now and then, and their outputs then say
# little about either.)  Served tokens are compared too: a trained model is mostly sure of its next token, random weights
# never are, so the model that serves has an output head of its own, the embedding moved on by one row.
MODELS = {"qwen2-0.5b": QWEN_05B, "qwen2-1.5b": QWEN_15B, "qwen2-0.5b-sure": dict(QWEN_05B, tie_word_embeddings=False), "lasizen": _lasizen(),
          "zodosun": _zodosun()}
MOST_STEP_TOKENS = 4096         # tokens of prompts in one step of a session
SEED = 7                        # of the models' weights: a model is a file, the seed of a state is its prompts'


def _vocab(model):
    c = MODELS[model]
    return c["vocab"] if "vocab" in c else c["vocab_size"]


def _write(folder, model):
    from easy_gpt.cpp_b200.weights import lasizen_init, random_init, safetensors_io, zodosun_init

    if model != "qwen2-0.5b-sure":
        {"lasizen": lasizen_init, "zodosun": zodosun_init}.get(model, random_init).write_random_model(folder, MODELS[model], SEED)
        return
    tensors = dict(random_init.random_tensors(MODELS[model], SEED))
    tensors["model.embed_tokens.weight"] *= 50.0                         # of order one, as the layers' sum
    tensors["lm_head.weight"] = tensors["model.embed_tokens.weight"].roll(1, 0)
    (folder / "config.json").write_text(json.dumps(MODELS[model]))
    safetensors_io.write_safetensors(folder / "model.safetensors", tensors.items())


@functools.lru_cache(maxsize=None)
def _folder(model):
    """A folder with the model's config.json and random weights, written once on a machine."""
    base = Path(tempfile.gettempdir()) / f"easy_gpt_perf_{os.getuid()}"
    folder = base / f"{model}_{SEED}"
    if not (folder / "model.safetensors").is_file():
        base.mkdir(parents=True, exist_ok=True)
        made = Path(tempfile.mkdtemp(dir=base))
        _write(made, model)
        try:
            made.rename(folder)
        except OSError:                                     # another process was first
            shutil.rmtree(made)
    return folder


@functools.lru_cache(maxsize=None)
def _runner(model, dtype):
    from easy_gpt.cpp_b200.native import NativeStepRunner

    tokens = 4096 if dtype == "float32" else 24576
    return NativeStepRunner(_folder(model), dtype, page_size=64, num_pages=tokens // 64 + 32, max_slots=32, max_tokens_per_request=8192)


@functools.lru_cache(maxsize=None)
def _engine(model):
    from easy_gpt.cpp_b200.native import NativeEngine

    return NativeEngine(_folder(model), cache_tokens=64 * 1024, max_active=64, max_tokens_per_request=4352)


# ---- cases ----------------------------------------------------------------------------------------------------------
def _session(model, batch, prompt, new, dtype="bfloat16"):
    return {"kind": "session", "model": model, "dtype": dtype, "batch": batch, "prompt": prompt, "new": new}


def _serve(model, batch, prompt, new):
    return {"kind": "serve", "model": model, "dtype": "bfloat16", "batch": batch, "prompt": prompt, "new": new}


def listed():
    return [
        # one user's short question: every token waits for the step before it, so latency and launches are all there is
        dict(_session("qwen2-0.5b", 1, 37, 31), name="chat_b1"),
        # a few conversations at once
        dict(_session("qwen2-0.5b", 8, 250, 24), name="chat_b8"),
        # a document to be scored or to be answered about: one long prompt, its last logits
        dict(_session("qwen2-0.5b", 1, 2048, 0), name="prompt_2048"),
        # a handful of prompts of odd lengths in one step, a few tokens for each: extraction, classification
        dict(_session("qwen2-0.5b", 5, 777, 3), name="prompts_ragged"),
        # the headline of the benchmark: eight requests deep in their contexts
        dict(_serve("qwen2-0.5b-sure", 8, 3800, 64), name="serve_b8_long"),
        # a busy server: 64 requests, prompts in portions beside decoding requests
        dict(_serve("qwen2-0.5b-sure", 64, 500, 64), name="serve_b64"),
        # the larger model of the family with a full batch
        dict(_session("qwen2-1.5b", 16, 120, 24), name="chat_15b_b16"),
        # the 32-bit path: what a port or a quantised model is checked against, logit by logit
        dict(_session("qwen2-0.5b", 4, 100, 8, "float32"), name="replay_f32"),
        # the further kinds of layers: a batch of prompts and the tokens behind them
        dict(_session("lasizen", 8, 256, 24), name="lasizen_b8"),
        dict(_session("zodosun", 8, 256, 24), name="zodosun_b8"),
        # and a long prompt with an odd length through one of them
        dict(_session("zodosun", 1, 2047, 1), name="zodosun_2047"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def draw(rng):
    kind = rng.choice(["qwen", "qwen", "qwen", "serve", "serve", "float32", "lasizen", "zodosun", "1.5b"])
    if kind == "serve":
        batch = _log_uniform(rng, 4, 64)
        return _serve("qwen2-0.5b-sure", batch, _log_uniform(rng, 24, min(3800, 32000 // batch)), rng.randint(16, 64))
    if kind == "float32":
        batch = _log_uniform(rng, 1, 6)
        return _session("qwen2-0.5b", batch, _log_uniform(rng, 3, 400 // batch), rng.randint(1, 8), "float32")
    if kind == "1.5b":
        batch = _log_uniform(rng, 1, 16)
        return _session("qwen2-1.5b", batch, _log_uniform(rng, 8, 1920 // batch), rng.randint(2, 24))
    batch = _log_uniform(rng, 1, 16)
    if kind == "qwen":
        return _session("qwen2-0.5b", batch, _log_uniform(rng, 5, min(4000, 8000 // batch)), rng.randint(0, 31))
    return _session(kind, batch, _log_uniform(rng, 5, 2048 // batch), rng.randint(1, 24))


def _lengths(case):
    """Prompt lengths of a batch: from the longest down to about half of it."""
    n, longest = case["batch"], case["prompt"]
    return [max(1, longest - i * longest // (2 * n)) for i in range(n)]


def _prompt_steps(lengths):
    """Steps of (request, first token, behind the last): prompts packed into steps, cut where a step is full."""
    steps, room = [[]], MOST_STEP_TOKENS
    for i, n in enumerate(lengths):
        at = 0
        while at < n:
            if room == 0:
                steps.append([])
                room = MOST_STEP_TOKENS
            take = min(room, n - at)
            steps[-1].append((i, at, at + take))
            at += take
            room -= take
    return steps


def _tokens(case, seed):
    rng = np.random.default_rng([seed, case["batch"], case["prompt"], case["new"]])
    extra = case["new"] if case["kind"] == "session" else 0
    return [rng.integers(0, _vocab(case["model"]), size=n + extra).tolist() for n in _lengths(case)]


def prepare(case, seed):
    state = {"case": case, "tokens": _tokens(case, seed), "lengths": _lengths(case)}
    if case["kind"] == "serve":
        state["engine"] = _engine(case["model"])
    else:
        state["runner"] = _runner(case["model"], case["dtype"])
        state["steps"] = _prompt_steps(state["lengths"])
    return state


def run(state):
    case, tokens, lengths = state["case"], state["tokens"], state["lengths"]
    if case["kind"] == "serve":
        return np.asarray(state["engine"].generate(tokens, max_new_tokens=case["new"], greedy=True))
    runner, logits = state["runner"], []
    for step in state["steps"]:
        rows = runner.run([(i, tokens[i][a:b], [b - a - 1] if b == lengths[i] else []) for i, a, b in step])
        if rows is not None:
            logits.append(rows)
    for s in range(case["new"]):
        logits.append(runner.run([(i, [tokens[i][n + s]], [0]) for i, n in enumerate(lengths)]))
    for i in range(case["batch"]):
        runner.end(i)
    return logits


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _layers_run(c):
    loop, n = c.get("loop"), len(c["layers"])
    return list(range(n)) if not loop else list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))


def _layer_sizes(c, layer):
    """(weights, cached values a token, operations per (query, key) pair) of a layer"""
    d, m = c["width"], layer["mixer"]
    ff = (2 if c["architecture"] == "Lasizen" else 3) * d * layer["mlp"]["ff"]
    if layer["type"] == "attention":
        H, G, k = m["heads"], m["kv_heads"], m["dim"]
        return 2 * d * (H + G) * k + ff, 2 * G * k, 4 * H * k
    if layer["type"] == "delta":
        H, G, k = m["heads"], m["kv_heads"], m["dim"]
        return d * (3 * H + 2 * G) * k + 2 * d * H + ff, 0, 0
    if layer["type"] == "general_delta":
        n = m["heads"] * m["dim"]
        return 6 * n * d + m["rank"] * (d + n) + ff, 0, 0
    l, r = m["left"], m["right"]
    w = d * (2 * l["heads"] * l["dim"] + 2 * l["kv_heads"] * l["dim"]) + 5 * d * r["heads"] * r["dim"]
    return w + ff, 2 * l["kv_heads"] * l["dim"], 4 * l["heads"] * l["dim"]


def work(case):
    """Every weight read once a step, every cached row read once by every decode step and written once, and the
    products of every token."""
    c, lengths, new, B = MODELS[case["model"]], _lengths(case), case["new"], case["batch"]
    size = 4 if case["dtype"] == "float32" else 2
    decodes = new if case["kind"] == "session" else new - 1             # the last token served is not run
    prompts = [sum(b - a for _, a, b in s) for s in _prompt_steps(lengths)] if case["kind"] == "session" else \
        [min(2048, sum(lengths) - at) for at in range(0, sum(lengths), 2048)]
    ran = prompts + [B] * decodes
    rows = B * (1 + decodes)
    pairs = sum((n + decodes) * (n + decodes + 1) / 2 for n in lengths)
    reads = sum(decodes * n + decodes * (decodes + 1) / 2 for n in lengths)
    total = sum(ran)
    if "vocab_size" in c:
        d, L, H, G = c["hidden_size"], c["num_hidden_layers"], c["num_attention_heads"], c["num_key_value_heads"]
        vocab, hd = c["vocab_size"], d // H
        once, cached, pair = L * (2 * d * (H + G) * hd + 3 * d * c["intermediate_size"]), L * 2 * G * hd, L * 4 * H * hd
    else:
        d, vocab = c["width"], c["vocab"]
        once, cached, pair = (sum(s) for s in zip(*(_layer_sizes(c, c["layers"][i]) for i in _layers_run(c))))
    head = d * vocab
    weights, flops = once * len(ran), 2 * once * total + pair * pairs
    weights += head * (1 + decodes)
    flops += 2 * head * rows
    result = rows * vocab * 4 if case["kind"] == "session" else B * new * 8
    return {"bytes": size * (weights + cached * (reads + total)) + result + 4 * total, "flops": flops}


def tolerance(case):
    if case["kind"] == "serve":
        return {"differ": 0.01}
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5}          # 3e-6 off the 64-bit result
    return {"rel": 3e-2}                # 0.7e-2 (zodosun) to 2e-2 (28 layers of 1.5b) off the 64-bit result


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------
class _Weights:
    """The tensors of a model folder, handed out in 64 bits on the GPU."""

    def __init__(self, folder):
        raw = np.memmap(folder / "model.safetensors", dtype=np.uint8, mode="r")
        (n,) = struct.unpack("<Q", bytes(raw[:8]))
        self.header = json.loads(bytes(raw[8:8 + n]))
        self.raw, self.at, self.held = raw, 8 + n, {}

    def __getitem__(self, name):
        if name not in self.held:
            h = self.header[name]
            assert h["dtype"] == "BF16"
            lo, hi = h["data_offsets"]
            bits = torch.from_numpy(np.array(self.raw[self.at + lo:self.at + hi])).view(torch.bfloat16)
            self.held[name] = bits.reshape(h["shape"]).cuda()
        return self.held[name].double()


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _seen(L, device):
    return torch.ones(L, L, dtype=torch.bool, device=device).tril()


def _halves(x, c, s, dims):
    """Value i of the first dims turned with value i + dims/2; c and s broadcast against x[..., :dims/2]."""
    a, b = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


def _angles(L, dims, base):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    return torch.arange(L, dtype=torch.float64, device="cuda")[:, None] * f


def _grouped(q, k, v, weigh):
    """Per request and head: weigh(scores) @ v; q [B, L, H, e], k and v [B, L, G, .]"""
    B, L, H, _ = q.shape
    group = H // k.shape[2]
    out = []
    for b in range(B):
        kb, vb = (t[b].permute(1, 0, 2).repeat_interleave(group, 0) for t in (k, v))
        out.append((weigh(q[b].permute(1, 0, 2) @ kb.transpose(1, 2)) @ vb).permute(1, 0, 2))
    return torch.stack(out).reshape(B, L, -1)


def _qwen_hidden(c, w, tokens):
    d, H, G = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"]
    hd, eps = d // H, c["rms_norm_eps"]
    x = w["model.embed_tokens.weight"][tokens]
    B, L = tokens.shape
    a = _angles(L, hd, c["rope_theta"])
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    hide = ~_seen(L, x.device)
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w[p + "input_layernorm.weight"]
        q, k, v = (h @ w[f"{p}self_attn.{n}_proj.weight"].T + w[f"{p}self_attn.{n}_proj.bias"] for n in "qkv")
        q, k = _halves(q.view(B, L, H, hd), cos, sin, hd), _halves(k.view(B, L, G, hd), cos, sin, hd)
        o = _grouped(q, k, v.view(B, L, G, hd), lambda s: (s * hd ** -0.5).masked_fill(hide, -math.inf).softmax(-1))
        x = x + o @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, eps) * w[p + "post_attention_layernorm.weight"]
        g = torch.nn.functional.silu(h @ w[p + "mlp.gate_proj.weight"].T)
        x = x + (g * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return _rms(x, eps) * w["model.norm.weight"]


def _qwen_head(c, w, y):
    return y @ w["model.embed_tokens.weight"].T


def _conv(x, taps):
    """A causal convolution over time on each channel; the last tap weighs the current token."""
    K, L = taps.shape[1], x.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, K - 1, 0))
    return sum(padded[:, j:j + L] * taps[:, j] for j in range(K))


def _lasizen_hidden(c, w, tokens):
    eps, F = c["norm"]["eps"], torch.nn.functional
    x = w["embed"][tokens] * c["embedding"]["scale"]
    B, L, d = x.shape
    at = torch.arange(L, device="cuda")

    def attention(h, p, m):
        H, G, k, rot, size = m["heads"], m["kv_heads"], m["dim"], m["rot"], m["mask"]["size"]
        sc, dims = rot["scaling"], rot["dims"]
        turn = lambda t: dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(rot["base"]))  # noqa: E731
        lo, hi = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=torch.float64, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        a = _angles(L, dims, rot["base"]) * (ramp / sc["factor"] + 1 - ramp)
        grow = 0.1 * math.log(sc["factor"]) + 1.0
        cos, sin = (a.cos() * grow)[:, None], (a.sin() * grow)[:, None]
        q, key = (_rms(_halves((h @ w[p + n].T).view(B, L, heads, k), cos, sin, dims), eps) for n, heads in (("q", H), ("k", G)))
        behind = at[:, None] - at
        hide = (behind < 0) | (behind >= size)

        def weigh(s):
            s = (s * m["scale"]).masked_fill(hide, -math.inf)
            return torch.cat([s, torch.zeros_like(s[..., :1])], -1).softmax(-1)[..., :-1]

        return _grouped(q, key, (h @ w[p + "v"].T).view(B, L, G, -1), weigh) @ w[p + "o"].T

    def delta(h, p, m):
        H, G, k, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, key, v = (F.silu(_conv(h @ w[p + n].T, w[p + n + ".conv"])) for n in "qkv")
        q, key = (t.view(B, L, G, k) / (t.view(B, L, G, k).square().sum(-1, keepdim=True) + 1e-6).sqrt() for t in (q, key))
        q, key = (t.repeat_interleave(H // G, 2) for t in (q * k ** -0.5, key))
        v = v.view(B, L, H, dv)
        beta = (h @ w[p + "b"].T).sigmoid()[..., None, None]
        decay = (-w[p + "A_log"].exp() * F.softplus(h @ w[p + "a"].T + w[p + "dt_bias"])).exp()[..., None, None]
        S, out = torch.zeros(B, H, k, dv, dtype=x.dtype, device=x.device), torch.empty_like(v)
        for t in range(L):
            S = decay[:, t] * S
            S = S + key[:, t, ..., None] * (beta[:, t] * (v[:, t, :, None] - key[:, t, :, None] @ S))
            out[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
        y = _rms(out, eps) * w[p + "norm"] * F.silu(h @ w[p + "g"].T).view(B, L, H, dv)
        return y.flatten(2) @ w[p + "o"].T

    for i in _layers_run(c):
        layer, p = c["layers"][i], f"l{i}."
        h = _rms(x, eps) * w[p + "norm1"]
        h = h + (F.pad(h, (0, 0, 1, 0))[:, :L] - h) * w[p + "shift"]
        x = x + _rms((attention if layer["type"] == "attention" else delta)(h, p + "mix.", layer["mixer"]), eps) * w[p + "norm1b"]
        z = (_rms(x, eps) * w[p + "norm2"]) @ w[p + "mlp.up"].T
        above, below = F.softplus(w[p + "mlp.act"])
        low = z.clamp(max=0)
        z = torch.where(z > 0, above * z * z + 0.5 * z, (0.5 + below) * (torch.expm1(low) - low) + 0.5 * low)
        x = x + _rms(z @ w[p + "mlp.down"].T, eps) * w[p + "norm2b"]
    return _rms(x, eps) * w["final.norm"]


def _plain_head(c, w, y):
    return y @ w["head"].T * c.get("logit_scale", 1.0)


def _zodosun_hidden(c, w, tokens):
    eps, groups, silu = c["norm"]["eps"], c["norm"]["groups"], torch.nn.functional.silu
    x = w["embed"][tokens]
    B, L, d = x.shape
    norm = lambda x, gain: _rms(x.view(B, L, groups, d // groups), eps).view(B, L, d) * gain  # noqa: E731
    a = torch.arange(L, dtype=torch.float64, device="cuda")[:, None] * 10000.0 ** (-2.0 * (torch.arange(d, device="cuda").double() // 2) / d)
    x = x + torch.where(torch.arange(d, device="cuda") % 2 == 0, a.sin(), a.cos())
    seen = _seen(L, x.device)

    def bucket(n, rows, most):
        half = rows // 2
        return n if n < half else min(rows - 1, half + math.floor(math.log(n / half) / math.log(most / half) * (rows - half)))

    def sigmoids(h, p, m):
        H, G, k, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q = _rms(h @ w[p + "q"].T + w[p + "q.b"], eps) * w[p + "q.norm"]
        key = _rms(h @ w[p + "k"].T + w[p + "k.b"], eps) * w[p + "k.norm"]
        v = (h @ w[p + "v"].T + w[p + "v.b"]).view(B, L, G, dv)
        temp = torch.tensor([1 + m["q_temp"]["coef"] * math.log((t + 1) // m["q_temp"]["every"] + 1) for t in range(L)], dtype=torch.float64, device="cuda")
        table = w[p + "rel"]
        by = table[[bucket(n, table.shape[0], m["bias_max"]) for n in range(L)]]
        at = torch.arange(L, device="cuda")
        bias = by[(at[:, None] - at).clamp(min=0)].permute(2, 0, 1) + w[p + "pb"][:, None, None]
        o = _grouped((q * temp[:, None]).view(B, L, H, k), key.view(B, L, G, k), v, lambda s: (s * m["scale"] + bias).sigmoid() * seen)
        return (o.view(B, L, H, dv) * (h @ w[p + "g"].T).sigmoid()[..., None]).flatten(2) @ w[p + "o"].T

    def fading(h, p, m):
        H, k, dv = m["heads"], m["dim"], m["vdim"]
        q, key, v = (silu(h @ w[p + n].T).view(B, L, H, -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")
        at = torch.arange(L, device="cuda")
        fade = decay[:, None, None] ** (at[:, None] - at).clamp(min=0) * seen
        y = _grouped(q, key, v, lambda s: s * fade)
        return (_rms(y, eps) * w[p + "norm"] * (h @ w[p + "g"].T).sigmoid()) @ w[p + "o"].T

    def delta(h, p, m):
        H, k = m["heads"], m["dim"]
        r, key, v = ((h @ w[p + n].T).view(B, L, H, k) for n in "rkv")
        decay = (-math.exp(-0.5) * ((h @ w[p + "w1"].T).tanh() @ w[p + "w2"].T + w[p + "w0"]).sigmoid()).exp().view(B, L, H, k)
        rate = (h @ w[p + "a"].T + w[p + "a.b"]).sigmoid().view(B, L, H, k)
        u = key / ((key * key).sum(-1, keepdim=True) + 1e-6).sqrt()
        S, out = torch.zeros(B, H, k, k, dtype=x.dtype, device=x.device), torch.empty_like(r)
        for t in range(L):
            held = u[:, t, :, None] @ S
            S = decay[:, t, ..., None] * S - (rate[:, t] * u[:, t])[..., None] * held + key[:, t, ..., None] * v[:, t, :, None]
            out[:, t] = (r[:, t, :, None] @ S)[:, :, 0]
        y = _rms(out, eps).reshape(B, L, H * k) * w[p + "norm"] * (h @ w[p + "g"].T).sigmoid()
        return y @ w[p + "o"].T

    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        h = norm(x, w[p + "norm1"])
        if layer["type"] == "general_delta":
            x = x + delta(h, p + "mix.", m)
        else:
            q = p + "mix."
            x = x + 0.5 * (_rms(sigmoids(h, q + "left.", m["left"]), eps) * w[q + "left.out"] + _rms(fading(h, q + "right.", m["right"]), eps) * w[q + "right.out"])
        h = norm(x, w[p + "norm2"])
        x = x + (silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
    return norm(x, w["final.norm"])


_PLAIN = {"lasizen": (_lasizen_hidden, _plain_head), "zodosun": (_zodosun_hidden, _plain_head)}


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "serve":
        return None                     # tokens: each hangs off the choices in front of it
    c, lengths, tokens = MODELS[case["model"]], _lengths(case), _tokens(case, seed)
    w = _Weights(_folder(case["model"]))
    hidden, head = _PLAIN.get(case["model"], (_qwen_hidden, _qwen_head))
    B, longest, new = case["batch"], max(len(t) for t in tokens), case["new"]
    padded = torch.tensor([t + [0] * (longest - len(t)) for t in tokens], device="cuda")        # causal: what stands behind a request does not matter
    y = torch.stack([y[n - 1:n + new] for y, n in zip(hidden(c, w, padded), lengths)])
    out = []
    for step in _prompt_steps(lengths):
        ends = [i for i, _, b in step if b == lengths[i]]
        if ends:
            out.append(head(c, w, y[ends, 0]).cpu().numpy())
    return out + [head(c, w, y[:, 1 + s]).cpu().numpy() for s in range(new)]
