"""What the engine is timed on: steps of a serving engine, and the sampler behind them.

A step case is one call of the step function, `ModelRunner.step`, on a batch of requests that the engine holds: `decoding`
requests whose contexts lie evenly between `context_lo` and `context_hi` tokens and that bring their newest token, beside
`portions` requests that bring `tokens` tokens of their prompts behind `behind` tokens that earlier steps put into the cache.
It returns the logits of every decoded token and of every portion's last token.  The models have the layer sizes of bench.py
at full depth, with random weights in the distribution its benchmarks use.  `prepare` builds the engine, lets it run the
requests up to the step, and repeats the step until its CUDA graph exists, as `LLMEngine.warm_up` does for a server; the step
can be repeated because it writes the same keys and values to the same slots.

A sampling case is the draw behind a step: `rows` rows of logits, one request each, with the options of `SamplingParams`.

The range that `draw` covers: 1 to 160 decoding requests with contexts of 16 to 4,096 tokens; portions of 16 to 4,096 tokens,
up to four in a step, behind up to 4,096 tokens; the two mixed; bfloat16 on the three layer sizes (the largest of them with
up to 16 decoding requests and 3,072 tokens), float32 on the smallest; 1 to 160 rows to sample.
"""

from __future__ import annotations

import json
import math
import os
import tempfile

import torch

from paged_llm_b200 import LLMEngine, SamplingParams
from paged_llm_b200.config.registry import parse_model_config
from paged_llm_b200.engine import Sequence, StepItem
from paged_llm_b200.sampling.sampler import Sampler
from paged_llm_b200.weights import write_random_stub

SIZES = {
    "tinyllama-1.1b": dict(vocab_size=32000, hidden_size=2048, intermediate_size=5632, num_hidden_layers=22,
                           num_attention_heads=32, num_key_value_heads=4, head_dim=64, rope_theta=10000.0,
                           rms_norm_eps=1e-5, tie_word_embeddings=False, max_position_embeddings=2048),
    "llama-3.2-1b": dict(vocab_size=128256, hidden_size=2048, intermediate_size=8192, num_hidden_layers=16,
                         num_attention_heads=32, num_key_value_heads=8, head_dim=64, rope_theta=500000.0,
                         rope_scaling=dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                           original_max_position_embeddings=8192),
                         rms_norm_eps=1e-5, tie_word_embeddings=True, max_position_embeddings=8192),
    "llama-3-8b": dict(vocab_size=128256, hidden_size=4096, intermediate_size=14336, num_hidden_layers=32,
                       num_attention_heads=32, num_key_value_heads=8, head_dim=128, rope_theta=500000.0,
                       rms_norm_eps=1e-5, tie_word_embeddings=False, max_position_embeddings=8192),
}
TINY, SMALL, LARGE = SIZES
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
BLOCK_SIZE = 16


def _step(name, model, dtype="bfloat16", decoding=0, context_lo=0, context_hi=0, portions=0, tokens=0, behind=0):
    case = {"kind": "step", "model": model, "dtype": dtype, "decoding": decoding, "context_lo": context_lo,
            "context_hi": context_hi, "portions": portions, "tokens": tokens, "behind": behind}
    return {"name": name, **case} if name else case


def _sample(name, rows, vocab, temperature, top_k, top_p):
    case = {"kind": "sample", "rows": rows, "vocab": vocab, "temperature": temperature, "top_k": top_k, "top_p": top_p}
    return {"name": name, **case} if name else case


def listed():
    return [
        # one user's chat: the latency of a token
        _step("decode-1", TINY, decoding=1, context_lo=640, context_hi=640),
        # the headline benchmark: eight requests of 512 prompt tokens in the middle of 256 decoded ones
        _step("decode-8", TINY, decoding=8, context_lo=640, context_hi=640),
        # a busy server of a small model
        _step("decode-64", TINY, decoding=64, context_lo=640, context_hi=640),
        # requests that arrived at different times, an odd number of them, some far into a long conversation
        _step("decode-ragged-27", SMALL, decoding=27, context_lo=131, context_hi=3500),
        # many short requests
        _step("decode-131", TINY, decoding=131, context_lo=70, context_hi=777),
        # a few users of a larger model
        _step("decode-8-8b", LARGE, decoding=8, context_lo=1031, context_hi=1279),
        # the first token of a short question
        _step("prompt-61", TINY, portions=1, tokens=61),
        # the first token behind a full token budget: the prefill benchmark
        _step("prompt-2048", TINY, portions=1, tokens=2048),
        # a long document for the larger model, in one step
        _step("prompt-8192-8b", LARGE, portions=1, tokens=8192),
        # chunked prefill beside decoding: two prompts continue while others decode
        _step("mixed-33", SMALL, decoding=33, context_lo=128, context_hi=1500, portions=2, tokens=389, behind=1024),
        # the 32-bit validation run: a few requests decode while a prompt comes in
        _step("float32-mixed", TINY, "float32", decoding=3, context_lo=100, context_hi=300, portions=1, tokens=125),
        # the draw for a full batch of a large vocabulary with every filter on
        _sample("sample-64", 64, 128256, 0.7, 50, 0.9),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prompt", "prompt", "mixed", "float32", "sample"))
    if kind == "sample":
        vocab = SIZES[rng.choice((TINY, SMALL))]["vocab_size"]
        return _sample(None, _log(rng, 1, 160), vocab, rng.choice((0.0, 0.6, 0.7, 1.0)), rng.choice((-1, 20, 50)),
                       rng.choice((1.0, 0.9, 0.95)))
    if kind == "float32":
        lo = _log(rng, 16, 400)
        many = rng.randint(0, 1)
        return _step(None, TINY, "float32", rng.randint(1, 5), lo, lo + rng.randint(0, 100), many, many * _log(rng, 16, 160))
    model = rng.choice((TINY, TINY, SMALL, SMALL, LARGE))
    if kind == "prompt":
        many = rng.choice((1, 1, 2, 4))
        longest = 2048 if model == TINY else 3072 if model == LARGE else 4096
        tokens = _log(rng, 16, longest // many)
        behind = 0 if rng.random() < 0.6 else _log(rng, 16, longest - tokens) if tokens + 16 < longest else 0
        return _step(None, model, portions=many, tokens=tokens, behind=behind)
    many = _log(rng, 1, 16 if model == LARGE else 160)
    longest = min({TINY: 2000, SMALL: 4000, LARGE: 3000}[model], 80000 // many)
    a, b = _log(rng, 16, longest), _log(rng, 16, longest)
    if kind == "decode":
        return _step(None, model, decoding=many, context_lo=min(a, b), context_hi=max(a, b))
    return _step(None, model, decoding=min(many, 63), context_lo=min(a, b), context_hi=max(a, b), portions=rng.choice((1, 1, 2)),
                 tokens=_log(rng, 16, 1500), behind=rng.choice((0, 0, 256)))


# ---- inputs -------------------------------------------------------------------------------------

def _contexts(case):
    """Tokens of each decoding request that are in the cache before the step (its newest token is not)."""
    n, lo, hi = case["decoding"], case["context_lo"], case["context_hi"]
    lens = [lo + (hi - lo) * i // max(1, n - 1) for i in range(n)]
    return [lens[(i * 7) % n] for i in range(n)] if n % 7 else lens       # long and short ones side by side


def _hf_config(case):
    return {"architectures": ["LlamaForCausalLM"], **SIZES[case["model"]]}


def _weights(case, seed):
    """Tensor name -> weights on the GPU: matrices N(0, 0.02), norm weights around one.  The projections that end a branch
    are divided by the root of the number of branches, and the embedding is of the size of their sum: the stream grows
    slowly, as it does in trained models, and rounding errors are not blown up layer by layer."""
    s, dtype = SIZES[case["model"]], DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, inner, d = s["hidden_size"], s["intermediate_size"], s["head_dim"]
    q, kv = s["num_attention_heads"] * d, s["num_key_value_heads"] * d

    def matrix(n, k, std=0.02):
        return torch.empty(n, k, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)

    def norm():
        return torch.empty(h, dtype=dtype, device="cuda").normal_(1.0, 0.05, generator=g)

    w = {"model.embed_tokens.weight": matrix(s["vocab_size"], h, 0.5), "model.norm.weight": norm()}
    if not s["tie_word_embeddings"]:
        w["lm_head.weight"] = matrix(s["vocab_size"], h)
    ends = 0.02 / (2 * s["num_hidden_layers"]) ** 0.5
    for i in range(s["num_hidden_layers"]):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = norm(), norm()
        for name, n, k in (("self_attn.q_proj", q, h), ("self_attn.k_proj", kv, h), ("self_attn.v_proj", kv, h),
                           ("self_attn.o_proj", h, q), ("mlp.gate_proj", inner, h), ("mlp.up_proj", inner, h),
                           ("mlp.down_proj", h, inner)):
            w[p + name + ".weight"] = matrix(n, k, ends if name in ("self_attn.o_proj", "mlp.down_proj") else 0.02)
    return w


def _requests(case, seed):
    """(token ids, how many of them the cache holds before the step) per request."""
    g = torch.Generator().manual_seed(seed + 1)
    lens = [(n + 1, n) for n in _contexts(case)] + [(case["behind"] + case["tokens"], case["behind"])] * case["portions"]
    vocab = SIZES[case["model"]]["vocab_size"]
    return [(torch.randint(0, vocab, (n,), generator=g).tolist(), held) for n, held in lens]


def _sample_inputs(case, seed):
    """Logits with a few likely tokens per row, as a trained model has them, and a stream per request."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    logits = torch.empty(case["rows"], case["vocab"], device="cuda").normal_(0.0, 2.5, generator=g)
    params = [SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=seed + i)
              for i in range(case["rows"])]
    return logits, [Sequence([1 + i], p) for i, p in enumerate(params)]


# ---- the measured calls -------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "sample":
        from paged_llm_b200.kernels.ops import CudaOps
        logits, seqs = _sample_inputs(case, seed)
        return {"sampler": Sampler(CudaOps("cuda"), seed), "logits": logits, "seqs": seqs}
    requests = _requests(case, seed)
    longest = max(len(ids) for ids, _ in requests)
    step_tokens = case["decoding"] + case["portions"] * case["tokens"]
    with tempfile.TemporaryDirectory() as folder:
        _, config = parse_model_config(_hf_config(case))
        write_random_stub(folder, config, seed=seed, dtype=case["dtype"])
        engine = LLMEngine(folder, dtype=case["dtype"], block_size=BLOCK_SIZE,
                           num_gpu_blocks=sum(-(-len(ids) // BLOCK_SIZE) for ids, _ in requests) + 16,
                           max_num_seqs=max(64, case["decoding"] + case["portions"]),
                           max_num_batched_tokens=max(2048, step_tokens), max_model_len=max(2048, longest + 16),
                           enable_prefix_caching=False)
    engine.model.load(_weights(case, seed))
    cache, runner = engine.block_manager, engine.runner
    items, pending = [], []

    def fill():
        runner.step(pending)
        for item in pending:
            item.seq.num_computed_tokens += item.num_new_tokens
        pending.clear()

    budget = 8192
    for ids, held in requests:
        seq = Sequence(ids, SamplingParams(temperature=0.0))
        if cache.allocate_slots(seq, len(ids)) is None:
            raise RuntimeError("the pool is too small for the case")
        if held:
            if sum(item.num_new_tokens for item in pending) + held > budget:
                fill()
            pending.append(StepItem(seq, held))
        items.append(StepItem(seq, len(ids) - held, (len(ids) - held - 1,)))
    if pending:
        fill()
    state = {"engine": engine, "items": items}
    for _ in range(3):
        run(state)
    return state


def run(state):
    if "sampler" in state:
        return state["sampler"].sample_on_device(state["logits"], state["seqs"])
    return state["engine"].runner.step(state["items"])


# ---- what a pass cannot do without --------------------------------------------------------------

def work(case):
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4.0 * n + 4.0 * case["rows"], "flops": 2.0 * n}
    s = SIZES[case["model"]]
    size = 2 if case["dtype"] == "bfloat16" else 4
    h, d, layers, vocab = s["hidden_size"], s["head_dim"], s["num_hidden_layers"], s["vocab_size"]
    q, kv = s["num_attention_heads"] * d, s["num_key_value_heads"] * d
    per_layer = h * (2 * q + 2 * kv + 3 * s["intermediate_size"])
    new = [(1, n) for n in _contexts(case)] + [(case["tokens"], case["behind"])] * case["portions"]
    tokens, rows = sum(t for t, _ in new), len(new)
    pairs = sum(t * held + t * (t + 1) // 2 for t, held in new)
    cached = sum(held for _, held in new)
    nbytes = size * (per_layer * layers + vocab * h + tokens * h + 2 * kv * layers * (cached + tokens)) + 4 * rows * vocab
    flops = 2.0 * tokens * per_layer * layers + 2.0 * rows * vocab * h + 4.0 * q * pairs * layers
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    """Relative errors as two correct implementations of the same precision show them: bfloat16 activations, keys, values
    and probabilities are rounded some ten times per layer, and two orders of summation round differently.  Measured between
    the few-token products and the library's on the same inputs: rel 0.006, max 0.034 at width 2,048; rel 0.016, max 0.073 at
    width 4,096; the distance of either from 64 bits is 0.0046 to 0.0054 and 0.014, and 2e-6 in float32."""
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.03, "max": 0.3} if case["model"] == LARGE else {"rel": 0.015, "max": 0.12}


# ---- the same in 64 bits ------------------------------------------------------------------------

def _angles(case, count):
    """cos and sin [count, head_dim / 2] in 64 bits."""
    s = SIZES[case["model"]]
    d, scaling = s["head_dim"], s.get("rope_scaling")
    freq = s["rope_theta"] ** (-torch.arange(0, d, 2, dtype=torch.float64, device="cuda") / d)
    if scaling:
        turns = scaling["original_max_position_embeddings"] * freq / (2 * math.pi)
        keep = ((turns - scaling["low_freq_factor"]) / (scaling["high_freq_factor"] - scaling["low_freq_factor"])).clamp(0, 1)
        freq = freq * (keep + (1 - keep) / scaling["factor"])
    angle = torch.arange(count, dtype=torch.float64, device="cuda")[:, None] * freq
    return angle.cos(), angle.sin()


def _attend(q, k, v, scale, q_rows):
    """Causal attention of the last `q_rows` positions, [heads, rows, d] against [kv heads, n, d]."""
    group, n = q.shape[0] // k.shape[0], k.shape[1]
    out = torch.empty_like(q)
    for j in range(k.shape[0]):
        for r in range(0, q_rows, 2048):
            e = min(q_rows, r + 2048)
            keys = n - q_rows + e
            p = q[j * group:(j + 1) * group, r:e] @ k[j, :keys].T * scale
            at = torch.arange(n - q_rows + r, n - q_rows + e, device="cuda")
            p.masked_fill_(torch.arange(keys, device="cuda") > at[:, None], -math.inf)
            out[j * group:(j + 1) * group, r:e] = torch.softmax(p, -1) @ v[j, :keys]
    return out


def exact(case, seed):
    if case["kind"] == "sample":
        return None                                   # the result is token ids, compared as they are
    s, requests = SIZES[case["model"]], _requests(case, seed)
    d, heads, kv = s["head_dim"], s["num_attention_heads"], s["num_key_value_heads"]
    lens = [len(ids) for ids, _ in requests]
    w = _weights(case, seed)
    cos, sin = _angles(case, max(lens))
    at = torch.cat([torch.arange(n, device="cuda") for n in lens])
    cos, sin = cos[at][:, None], sin[at][:, None]

    def wide(name):
        return w.pop(name).double()

    def normed(x, weight):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + s["rms_norm_eps"]) * weight

    def rotated(x):
        a, b = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    embed = w["model.embed_tokens.weight"]
    x = embed[torch.tensor([t for ids, _ in requests for t in ids], device="cuda")].double()
    for i in range(s["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = normed(x, wide(p + "input_layernorm.weight"))
        q = rotated((h @ wide(p + "self_attn.q_proj.weight").T).view(-1, heads, d)).transpose(0, 1)
        k = rotated((h @ wide(p + "self_attn.k_proj.weight").T).view(-1, kv, d)).transpose(0, 1)
        v = (h @ wide(p + "self_attn.v_proj.weight").T).view(-1, kv, d).transpose(0, 1)
        parts, o = [], 0
        for n in lens:
            parts.append(_attend(q[:, o:o + n], k[:, o:o + n], v[:, o:o + n], d ** -0.5, n))
            o += n
        h = torch.cat(parts, 1).transpose(0, 1).reshape(-1, heads * d)
        x += h @ wide(p + "self_attn.o_proj.weight").T
        h = normed(x, wide(p + "post_attention_layernorm.weight"))
        gate, up, down = (wide(f"{p}mlp.{m}_proj.weight").T for m in ("gate", "up", "down"))
        for r in range(0, h.shape[0], 8192):
            rows = h[r:r + 8192]
            x[r:r + 8192] += (torch.nn.functional.silu(rows @ gate) * (rows @ up)) @ down
    last = torch.tensor(lens, device="cuda").cumsum(0) - 1
    head = (embed if s["tie_word_embeddings"] else w["lm_head.weight"]).double()
    return normed(x[last], wide("model.norm.weight")) @ head.T
