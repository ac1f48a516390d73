"""Steps of 17 to 64 tokens of a decoder whose products hand rows prepared for the next norm from one to the next (csrc/gemm_batch.cu),
through the native step runner and against the plain model: decode steps (captured ones with padded rows among them), prompts, portions
beside decoded tokens, with all that stands around the chain (a first layer without prepared rows, windows, biases, gains, rows for the
head), the numbers of tokens next to where it ends, and models of which only a part fits."""
import numpy as np
import pytest

import engine_harness as H
import plain_model
import tiny_configs
from test_native_engine_gpu import BF16_REL, run_native
from test_schedules_gpu import trace_many_live

pytestmark = pytest.mark.gpu

# sizes that every product of the chain takes (multiples of 64, K of four stages and more)
TAKEN = {
    "architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2",
    "num_hidden_layers": 3, "hidden_size": 256, "num_attention_heads": 4, "num_key_value_heads": 2, "head_dim": 64,
    "intermediate_size": 512, "vocab_size": 384, "rope_theta": 10000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": False,
    "max_position_embeddings": 2048, "bos_token_id": -1, "eos_token_id": -1, "use_sliding_window": False,
}
CONFIGS = {
    "taken": TAKEN,
    "window, heads of 128, no biases": dict(TAKEN, num_attention_heads=2, num_key_value_heads=1, head_dim=128, attention_bias=False, use_sliding_window=True, sliding_window=40,
                                            max_window_layers=1),
    "gate and up refused": dict(TAKEN, intermediate_size=528),
    "down refused": dict(TAKEN, intermediate_size=160),
    "queries, keys and values refused": dict(TAKEN, num_attention_heads=8, head_dim=32),
}


def products(c):
    """(epilogue, N, K, head size) of a layer's products: queries, keys and values; into the residual twice; gate and up"""
    d, hd, ff = c["hidden_size"], c["head_dim"], c["intermediate_size"]
    heads, kv = c["num_attention_heads"], c["num_key_value_heads"]
    return [(3, (heads + 2 * kv) * hd, d, hd), (4, d, heads * hd, 0), (2, 2 * ff, d, 0), (4, d, ff, 0)]


@pytest.fixture(scope="module", params=list(CONFIGS))
def model(request, tmp_path_factory):
    from easy_gpt.cpp_b200 import kernels
    from easy_gpt.cpp_b200.weights.random_init import write_random_model

    c = CONFIGS[request.param]
    takes = [kernels.library().eg_gemm_batch_takes(*p) > 0 for p in products(c)]
    assert all(takes) == ("refused" not in request.param), takes
    folder = write_random_model(tmp_path_factory.mktemp("chain"), c, store_dtype="float32", seed=21, std=0.06, bias_std=0.1, gain_std=0.1)
    requests = {f"q{i}": tiny_configs.random_tokens(c["vocab_size"], 24 + (7 * i) % 40, 500 + i) for i in range(65)}
    cfg, w = plain_model.read_model_dir(folder, round_to_bf16=True)
    refs = {rid: plain_model.forward_logits(cfg, w, toks).numpy() for rid, toks in requests.items()}
    # (the bound of the native engine's replays; the library's products, in a step of 33 tokens, are up to 1.6e-2 off here)
    return folder, requests, refs, BF16_REL * max(float(np.abs(r).max()) for r in refs.values())


def check(model, steps, live, what):
    from easy_gpt.cpp_b200.native import NativeStepRunner

    folder, _, refs, tol = model
    runner = NativeStepRunner(folder, "bfloat16", 16, H.max_live_tokens(steps, 16) // 16, live)
    got = run_native(runner, steps)
    assert got
    H.compare(got, refs, tol, what)
    return runner


@pytest.mark.parametrize("live", [16, 17, 24, 32, 33, 48, 64, 65])
def test_decode_steps(model, live):
    """`live` requests one token each, again and again, one of them left out of every other step: buckets of a captured step with a padded row"""
    requests = dict(list(model[1].items())[:live])
    runner = check(model, trace_many_live(requests, decode_tokens=10, per_step=2, portion=64), live, f"{live} decoding")
    assert runner.info("graph_replays") >= 8


@pytest.mark.parametrize("length", [16, 17, 31, 32, 33])
def test_prompts(model, length):
    """Prompts of so many tokens alone in their steps, logits at each of them; then what is left of them"""
    steps = []
    for rid, toks in list(model[1].items())[:6]:
        first = min(length, len(toks) - 1)
        steps.append({"step": len(steps), "entries": [{"id": rid, "tokens": toks[:first], "want": list(range(first))}], "end": []})
        steps.append({"step": len(steps), "entries": [{"id": rid, "tokens": toks[first:], "want": [len(toks) - first - 1]}], "end": [rid]})
    check(model, steps, 2, f"prompts of {length}")


def test_portions_beside_decoded_tokens(model):
    """A portion of a prompt beside eleven decoding requests, 17 to 32 tokens in all; some rows are wanted"""
    requests = model[1]
    ids = list(requests)
    decoding, late = ids[:11], ids[11:16]
    steps = [{"step": 0, "entries": [{"id": r, "tokens": requests[r][:14], "want": [13]} for r in decoding], "end": []}]
    at = {r: 14 for r in decoding}
    for k, rid in enumerate(late):
        toks, done = requests[rid], 0
        while done < len(toks):
            n = min(6 + 3 * k, len(toks) - done)
            entries = [{"id": r, "tokens": [requests[r][at[r]]], "want": [0]} for r in decoding if at[r] < len(requests[r])]
            for e in entries:
                at[e["id"]] += 1
            entries.append({"id": rid, "tokens": toks[done:done + n], "want": [n - 1]})
            done += n
            steps.append({"step": len(steps), "entries": entries, "end": [rid] if done == len(toks) else []})
    steps[-1]["end"] = steps[-1]["end"] + decoding
    check(model, steps, 16, "portions")
