"""The work this engine is measured on: steps, prompts and generations through its public entry points.

A case names a model shape (random weights of that shape, drawn from the seed), the type it runs in, and what one
pass does:

* ``generate``  - ``Engine.generate``: prompts in, greedy tokens out, everything between them included;
* ``replay``    - the step function fed token by token and portion by portion, as ``bin/trace_run`` feeds it:
                  prompts in portions of ``chunk`` tokens beside the single tokens of requests that are further on;
* ``prompts``   - whole prompts in one step (prefill), logits at each prompt's end;
* ``chunked``   - one long prompt in portions of ``chunk`` tokens;
* ``decode``    - one token for each of ``batch`` requests that hold ``context`` tokens;
* ``mixed``     - one step of single tokens of ``batch`` requests beside a portion of a new prompt.

Requests that already hold tokens are given random keys and values of the deviation that random weights produce, in
place of prompts run through the model.  The large shapes run with their first 4 to 12 layers: every layer does the
same work, and through a random model's whole depth bfloat16 rounding alone grows to 3-5 % of the logits, which would
leave nothing to compare.  ``exact`` restates the decoders in float64 with plain torch and draws the
same weights with a restatement of the generator (the formulas in csrc/random_weights.h).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from aegean_tge_b200 import Engine
from aegean_tge_b200.bench_tools import mozepel_config
from aegean_tge_b200.engine.batch import Portion

QWEN2 = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "use_sliding_window": False, "hidden_act": "silu"}
# width, heads, kv heads, head size, gated inner width, vocabulary, layers, rotation base, eps, tied head, longest context
SHAPES = {
    "tiny-a": (64, 4, 2, 16, 176, 256, 2, 10000.0, 1e-6, True, 256),
    "tiny-b": (96, 3, 1, 32, 256, 384, 3, 1000000.0, 1e-5, False, 512),
    "1.5b": (1536, 12, 2, 128, 8960, 152064, 28, 1000000.0, 1e-6, False, 32768),
    "7b": (3584, 28, 4, 128, 18944, 152064, 28, 1000000.0, 1e-6, False, 32768),
    "14b": (5120, 40, 8, 128, 13824, 152064, 48, 1000000.0, 1e-6, False, 32768),
    "32b": (5120, 40, 8, 128, 27648, 152064, 64, 1000000.0, 1e-6, False, 32768),
}
ROOM = 512      # tokens a decoding request may gain before a new request of the same length takes its place


def listed():
    return [
        # the smallest calls: a few short prompts and sixteen tokens each on a model of a test's size
        {"name": "tiny-a-generate-f32", "kind": "generate", "design": "qwen2", "shape": "tiny-a", "layers": 2,
         "dtype": "float32", "page": 64, "lengths": "1,7,33", "new": 16},
        # a trace of ragged requests in small portions beside single tokens, logits wanted at every place that samples
        {"name": "tiny-b-replay-f32", "kind": "replay", "design": "qwen2", "shape": "tiny-b", "layers": 3,
         "dtype": "float32", "page": 16, "lengths": "5,19,64,130", "new": 24, "chunk": 16},
        # one user's generation: a step reads all weights for one token
        {"name": "7b-decode-b1", "kind": "decode", "design": "qwen2", "shape": "7b", "layers": 12, "dtype": "bfloat16",
         "page": 16, "batch": 1, "context": 2048},
        # a small batch, the benchmark's headline
        {"name": "7b-decode-b8", "kind": "decode", "design": "qwen2", "shape": "7b", "layers": 12, "dtype": "bfloat16",
         "page": 16, "batch": 8, "context": 2048},
        # a full batch: the cache's bytes count as much as half of the weights'
        {"name": "7b-decode-b64", "kind": "decode", "design": "qwen2", "shape": "7b", "layers": 12, "dtype": "bfloat16",
         "page": 64, "batch": 64, "context": 2048},
        # an ordinary long prompt
        {"name": "7b-prompt-2048", "kind": "prompts", "design": "qwen2", "shape": "7b", "layers": 12, "dtype": "bfloat16",
         "page": 16, "lengths": "2048"},
        # the first step of a few short chats that arrived together
        {"name": "7b-prompts-short", "kind": "prompts", "design": "qwen2", "shape": "7b", "layers": 12, "dtype": "bfloat16",
         "page": 64, "lengths": "23,61,109"},
        # continuous batching: requests of ragged lengths decode while a prompt arrives
        {"name": "14b-mixed", "kind": "mixed", "design": "qwen2", "shape": "14b", "layers": 8, "dtype": "bfloat16",
         "page": 64, "batch": 31, "context": 4096, "tokens": 1187},
        # a long prompt in portions on the widest layers
        {"name": "32b-chunked-8192", "kind": "chunked", "design": "qwen2", "shape": "32b", "layers": 4, "dtype": "bfloat16",
         "page": 64, "tokens": 8192, "chunk": 2048},
        # the float32 path that results are checked against: a prompt, and a step of a small batch
        {"name": "7b-prompt-512-f32", "kind": "prompts", "design": "qwen2", "shape": "7b", "layers": 4, "dtype": "float32",
         "page": 64, "lengths": "512"},
        {"name": "7b-decode-b8-f32", "kind": "decode", "design": "qwen2", "shape": "7b", "layers": 4, "dtype": "float32",
         "page": 64, "batch": 8, "context": 1000},
        # a design with recurrent state, sliding windows and pooled blocks: its prompt
        {"name": "mozepel-prompt-2048", "kind": "prompts", "design": "mozepel", "shape": "7b", "layers": 8,
         "dtype": "bfloat16", "page": 64, "lengths": "2048"},
    ]


def _spread(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["generate", "replay", "decode", "decode", "decode", "prompts", "prompts", "mixed", "chunked",
                       "decode-f32", "prompts-f32", "mozepel"])
    page = rng.choice([16, 64])
    if kind in ("generate", "replay"):
        shape = rng.choice(["tiny-a", "tiny-b"])
        lengths = ",".join(str(_spread(rng, 1, 130)) for _ in range(rng.randint(1, 6)))
        case = {"kind": kind, "design": "qwen2", "shape": shape, "layers": SHAPES[shape][6], "dtype": "float32",
                "page": page, "lengths": lengths, "new": rng.randint(4, 24)}
        if kind == "replay":
            case["chunk"] = rng.choice([8, 16, 33, 64])
        return case
    if kind == "mozepel":
        return {"kind": "prompts", "design": "mozepel", "shape": rng.choice(["1.5b", "7b"]), "layers": rng.choice([4, 8]),
                "dtype": "bfloat16", "page": page, "lengths": str(_spread(rng, 200, 3000))}
    f32 = kind.endswith("-f32")
    kind = kind.split("-")[0]
    shape = rng.choice(["1.5b", "7b"] if f32 else ["1.5b", "7b", "14b", "32b"])
    case = {"kind": kind, "design": "qwen2", "shape": shape, "layers": rng.randint(2, 4 if f32 else 8),
            "dtype": "float32" if f32 else "bfloat16", "page": page}
    if kind == "decode":
        case["batch"] = _spread(rng, 1, 12 if f32 else 64)
        case["context"] = _spread(rng, 30, 1500 if f32 else min(16000, 160000 // case["batch"]))
    elif kind == "prompts":
        case["lengths"] = ",".join(str(_spread(rng, 7, 500 if f32 else 2500)) for _ in range(1 if f32 else rng.randint(1, 3)))
    elif kind == "mixed":
        case["batch"], case["context"], case["tokens"] = rng.randint(1, 40), _spread(rng, 200, 4096), _spread(rng, 16, 2048)
    else:
        case["tokens"], case["chunk"] = _spread(rng, 2100, 8192), rng.choice([512, 1024, 2048])
    return case


# ----------------------------------------------------------------------------
# models, requests and their inputs
# ----------------------------------------------------------------------------
def config_of(case):
    width, heads, kv_heads, head_dim, inner, vocab, _layers, base, eps, tied, longest = SHAPES[case["shape"]]
    if case["design"] == "mozepel":
        return mozepel_config(width, heads, kv_heads, head_dim, inner, case["layers"], vocab)
    return dict(QWEN2, num_hidden_layers=case["layers"], hidden_size=width, num_attention_heads=heads,
                num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=inner, vocab_size=vocab,
                rope_theta=base, rms_norm_eps=eps, tie_word_embeddings=tied, max_position_embeddings=longest)


def token_ids(vocab, count, seed, which):
    rng = np.random.Generator(np.random.PCG64([seed, which]))
    return rng.integers(0, vocab, count).tolist()


def prompt_lengths(case):
    return [int(n) for n in case["lengths"].split(",")]


def held_lengths(case, seed):
    """How many tokens each request already holds: equal in ``decode``, ragged in ``mixed``."""
    if case["kind"] == "decode":
        return [case["context"]] * case["batch"]
    rng = random.Random(seed)
    return [rng.randint(min(128, case["context"]), case["context"]) for _ in range(case["batch"])]


def held_entries(case, seed, which, length):
    """The keys and values request ``which`` holds: [layers, kv heads, length, head size] each, in the run type."""
    width, _heads, kv_heads, head_dim = SHAPES[case["shape"]][:4]
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000 + which)
    shape = (case["layers"], kv_heads, length, head_dim)
    dtype = getattr(torch, case["dtype"])
    deviation = 0.02 * math.sqrt(width)        # of a product of a normed row with weights of deviation 0.02
    return tuple(torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(deviation).to(dtype)
                 for _ in range(2))


def replay_steps(case, tokens):
    """The trace: per step a list of (request, tokens, wanted places); a request samples from its prompt's end on."""
    lengths = prompt_lengths(case)
    done, steps = [0] * len(lengths), []
    while any(d < len(t) for d, t in zip(done, tokens)):
        step = []
        for r, length in enumerate(lengths):
            begin = done[r]
            if begin == len(tokens[r]):
                continue
            end = min(begin + case["chunk"], length) if begin < length else begin + 1
            step.append((r, tokens[r][begin:end], [end - begin - 1] if end >= length else []))
            done[r] = end
        steps.append(step)
    return steps


def case_tokens(case, seed):
    """The given token ids, one list per request (of ``mixed``, the new prompt last)."""
    vocab, kind = SHAPES[case["shape"]][5], case["kind"]
    if kind == "replay":
        counts = [n + case["new"] - 1 for n in prompt_lengths(case)]
    elif kind in ("generate", "prompts"):
        counts = prompt_lengths(case)
    elif kind == "chunked":
        counts = [case["tokens"]]
    elif kind == "decode":
        counts = [2] * case["batch"]           # one before the first pass, and the one every pass repeats
    else:
        counts = [1] * case["batch"] + [case["tokens"]]
    return [token_ids(vocab, count, seed, r) for r, count in enumerate(counts)]


def hold(engine, names, lengths, entries=None):
    """Admits requests that hold so many tokens; ``entries`` gives their keys and values."""
    cache = engine.cache
    for which, (name, length) in enumerate(zip(names, lengths)):
        cache.admit(name)
        cache.grow(name, length)
        cache.set_computed(name, length)
        if entries is None:
            continue
        pages = torch.tensor(cache.groups[0].tables[name], device="cuda")
        for tensor, rows in zip((cache.groups[0].storage["k"], cache.groups[0].storage["v"]), entries(which, length)):
            layers, kv_heads, _length, head_dim = rows.shape
            padded = torch.zeros((layers, kv_heads, len(pages) * cache.page_size, head_dim), dtype=rows.dtype, device="cuda")
            padded[:, :, :length] = rows
            tensor[:, pages] = padded.view(layers, kv_heads, len(pages), cache.page_size, head_dim).transpose(1, 2)


def prepare(case, seed):
    kind, page = case["kind"], case["page"]
    tokens = case_tokens(case, seed)
    held = held_lengths(case, seed) if kind in ("decode", "mixed") else []
    longest = [n + ROOM for n in held]
    if kind in ("generate", "replay"):
        longest += [n + case["new"] for n in prompt_lengths(case)]
    elif kind != "decode":
        longest += [len(t) for t in tokens[len(held):]]
    engine = Engine(random_config=config_of(case), seed=seed, dtype=case["dtype"], context=max(max(longest), 4096),
                    num_pages=sum(-(-n // page) for n in longest), max_batch_tokens=2048, max_requests=len(longest) + 1,
                    page_size=page)
    state = {"kind": kind, "engine": engine, "held": held, "names": [f"r{r}" for r in range(len(held))], "room": ROOM}
    if held:
        hold(engine, state["names"], held, lambda which, length: held_entries(case, seed, which, length))
    if kind == "generate":
        state["prompts"], state["new"] = tokens, case["new"]
    elif kind == "replay":
        state["steps"] = [[Portion(f"r{r}", part, want) for r, part, want in step] for step in replay_steps(case, tokens)]
    elif kind == "prompts":
        state["steps"] = [[Portion(f"p{r}", part, [len(part) - 1]) for r, part in enumerate(tokens)]]
    elif kind == "chunked":
        starts = range(0, case["tokens"], case["chunk"])
        parts = [tokens[0][begin:begin + case["chunk"]] for begin in starts]
        state["steps"] = [[Portion("p0", part, [len(part) - 1] if part is parts[-1] else [])] for part in parts]
    elif kind == "decode":
        state["room"] -= 1
        engine.runner.step([Portion(name, t[:1], [0]) for name, t in zip(state["names"], tokens)])
        state["portions"] = [Portion(name, t[1:], [0]) for name, t in zip(state["names"], tokens)]
    else:
        state["portions"] = [Portion(name, t, [0]) for name, t in zip(state["names"], tokens)]
        state["portions"].append(Portion("new", tokens[-1], [len(tokens[-1]) - 1]))
    torch.cuda.synchronize()
    return state


def run(state):
    engine, kind = state["engine"], state["kind"]
    if kind == "generate":
        return np.array(engine.generate(state["prompts"], n=state["new"]))
    if "steps" in state:
        logits = [engine.runner.step(step) for step in state["steps"]]
        for name in {portion.request for step in state["steps"] for portion in step}:
            engine.runner.finish(name)
        return [rows for rows in logits if rows is not None]
    if state["room"] == 0:                     # the requests are as long as they may get: new ones take their place
        for name in state["names"]:
            engine.runner.finish(name)
        hold(engine, state["names"], state["held"])
        state["room"] = ROOM
    state["room"] -= 1
    logits = engine.runner.step(state["portions"])
    if kind == "mixed":
        engine.runner.finish("new")
    return logits


# ----------------------------------------------------------------------------
# what a pass cannot do without, and how close two correct passes are
# ----------------------------------------------------------------------------
def work(case):
    """Every weight and every held key and value read once, every new one and the logits written once."""
    width, heads, kv_heads, head_dim, inner, vocab, _layers, _base, _eps, _tied, _longest = SHAPES[case["shape"]]
    element, layers, kind = 2 if case["dtype"] == "bfloat16" else 4, case["layers"], case["kind"]
    per_layer = width * head_dim * (2 * heads + 2 * kv_heads) + 3 * width * inner
    kv_token = 2 * kv_heads * head_dim * element * layers
    pairs_flops = 4 * heads * head_dim * layers            # per (query, key) pair: scores and their product with V
    triangle = lambda n: n * (n + 1) / 2
    if case["design"] == "mozepel":
        (n,) = prompt_lengths(case)
        windowed, decayed, half = layers // 4, layers - layers // 4, max(heads // 2, 1)
        matrices = (decayed * 5 * width * heads * head_dim + 3 * width * inner * layers
                    + windowed * (width * head_dim * (2 * heads + 2 * kv_heads) + width * half * (head_dim + 3 * head_dim)))
        near = triangle(n) - triangle(max(n - 1024, 0)) + triangle(max(n - 1024, 0)) / 64
        recurrence = 4 * n * head_dim * (decayed * heads * head_dim + windowed * half * head_dim // 2)
        return {"bytes": 2 * (matrices + vocab * width) + 4 * vocab,
                "flops": 2 * matrices * n + 2 * vocab * width + 4 * heads * head_dim * windowed * near + recurrence}
    if kind == "decode":
        rows, outputs, pairs, read = case["batch"], case["batch"], case["batch"] * case["context"], case["batch"] * case["context"]
    elif kind == "mixed":
        expected = case["batch"] * (min(128, case["context"]) + case["context"]) / 2
        rows, outputs, read = case["batch"] + case["tokens"], case["batch"] + 1, expected
        pairs = expected + triangle(case["tokens"])
    elif kind == "chunked":
        rows, outputs, pairs, read = case["tokens"], 1, triangle(case["tokens"]), 0
    else:
        lengths = prompt_lengths(case)
        new = case["new"] if kind in ("generate", "replay") else 1
        rows, outputs, read = sum(lengths) + len(lengths) * (new - 1), len(lengths) * new, 0
        pairs = sum(triangle(n + new - 1) for n in lengths)
    weights = (layers * per_layer + vocab * width) * element
    written = kv_token * rows + (4 * outputs * vocab if kind != "generate" else 8 * outputs)
    return {"bytes": weights + kv_token * read + written,
            "flops": 2 * rows * layers * per_layer + 2 * outputs * vocab * width + pairs_flops * pairs}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"                         # greedy tokens
    if case["dtype"] == "float32":
        return {"rel": 2e-5}                   # of float64: 4e-7 (tiny) to 2.1e-5 (angles of far positions in float32)
    # bfloat16 rounding anywhere in a layer moves all that follows: two attention kernels (other orders of summation) gave
    # logits 0.2 to 1.6 % apart at 4 to 12 layers and a largest difference of 0.04 to 0.09, both of them 1.1 to 2.5 % off float64
    return {"rel": 3e-2, "max": 0.35}


# ----------------------------------------------------------------------------
# the same in 64 bits
# ----------------------------------------------------------------------------
_MASK = (1 << 64) - 1
_GOLDEN = 0x9E3779B97F4A7C15


def _signed(z):
    return z - (1 << 64) if z >> 63 else z


def _mix_int(z):
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _MASK
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _MASK
    return z ^ (z >> 31)


def _shift(z, bits):
    return (z >> bits) & ((1 << (64 - bits)) - 1)          # a logical shift of int64


def _words(key, first, count, stride):
    counter = torch.arange(first + 1, first + 1 + count * stride, stride, dtype=torch.int64, device="cuda")
    z = counter.mul_(_signed(_GOLDEN)).add_(_signed(key))
    z = (z ^ _shift(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _shift(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _shift(z, 31)


class Weights:
    """Tensors of the random model by name: the engine's generator restated, rounded as the engine stores them."""

    def __init__(self, case, seed):
        self.seed, self.dtype = seed, getattr(torch, case["dtype"])

    def _key(self, name):
        h = 0xCBF29CE484222325
        for byte in name.encode("utf-8"):
            h = ((h ^ byte) * 0x100000001B3) & _MASK
        return _mix_int(h ^ _mix_int((self.seed + _GOLDEN) & _MASK))

    def normal(self, name, shape, std, matrix=True):
        key, total = self._key(name), math.prod(shape)
        scale = float(np.float32(std / (2.0 * math.sqrt(8.0 * (65536.0 ** 2 - 1.0) / 12.0))))
        out = torch.empty(total, dtype=torch.float64, device="cuda")
        step = 1 << 25
        for begin in range(0, total, step):
            count = min(step, total - begin)
            fields = torch.zeros(count, dtype=torch.int64, device="cuda")
            for odd in (0, 1):
                word = _words(key, 2 * begin + odd, count, 2)
                for field in range(4):
                    fields += (word >> (16 * field)) & 0xFFFF
            value = (2 * fields - 8 * 65535).to(torch.float32) * scale
            out[begin:begin + count] = value.to(self.dtype) if matrix else value
        return out.view(shape)

    def uniform(self, name, shape, lo, hi):
        base, span = round(lo * (1 << 24)), round((hi - lo) * (1 << 24))
        high = _shift(_words(self._key(name), 0, math.prod(shape), 1), 32)
        return (((high * span) >> 32) + base).to(torch.float64).mul_(2.0 ** -24).view(shape)


def _unit(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _rotate(x, positions, dims, frequencies):
    """x [T, heads, d]: number i < dims/2 is paired with number i + dims/2; the rest passes."""
    angle = positions.to(torch.float64)[:, None] * frequencies[None, :]
    cos, sin = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]
    lo, hi = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin, x[..., dims:]], dim=-1)


def _frequencies(dims, base, scaling=None):
    out = []
    for i in range(dims // 2):
        f = base ** (-2.0 * i / dims)
        if scaling is not None:
            wavelength = 2.0 * math.pi / f
            s = (scaling["original"] / wavelength - scaling["low"]) / (scaling["high"] - scaling["low"])
            s = min(max(s, 0.0), 1.0)
            f = (1.0 - s) * f / scaling["factor"] + s * f
        out.append(f)
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _attend(q, k, v, scale, start):
    """q [T, H, d] at positions start..., k and v [start + T, G, d]: causal attention, in blocks of queries."""
    heads, groups = q.shape[1], k.shape[1]
    k, v = (t.transpose(0, 1).repeat_interleave(heads // groups, dim=0) for t in (k, v))      # [H, C, d]
    out = torch.empty_like(q)
    for begin in range(0, q.shape[0], 512):
        part = q[begin:begin + 512].transpose(0, 1)
        last = start + begin + part.shape[1]
        scores = scale * (part @ k[:, :last].transpose(1, 2))
        at = torch.arange(start + begin, last, device="cuda")[:, None]
        scores.masked_fill_(torch.arange(last, device="cuda")[None, :] > at, -math.inf)
        out[begin:begin + 512] = (torch.softmax(scores, dim=-1) @ v[:, :last]).transpose(0, 1)
    return out


def qwen2_logits(case, weights, sequences, wanted, entries=None):
    """``sequences``: (first position, tokens) per request; ``wanted``: rows of all tokens joined.  Logits of those rows."""
    width, heads, kv_heads, head_dim, inner, vocab, _layers, base, eps, tied, _longest = SHAPES[case["shape"]]
    device = "cuda"
    ids = torch.tensor([t for _, tokens in sequences for t in tokens], device=device)
    x = weights.normal("model.embed_tokens.weight", (vocab, width), 0.02)[ids]
    freq = _frequencies(head_dim, base)
    positions = torch.cat([torch.arange(first, first + len(tokens), device=device) for first, tokens in sequences])
    held = [entries(r, first) if first else None for r, (first, _tokens) in enumerate(sequences)]
    for n in range(case["layers"]):
        p = f"model.layers.{n}."
        h = _unit(x, eps) * weights.uniform(p + "input_layernorm.weight", (width,), 0.9, 1.1)
        q, k, v = (h @ weights.normal(f"{p}self_attn.{t}_proj.weight", (rows * head_dim, width), 0.02).T
                   + weights.normal(f"{p}self_attn.{t}_proj.bias", (rows * head_dim,), 0.02, matrix=False)
                   for t, rows in (("q", heads), ("k", kv_heads), ("v", kv_heads)))
        q = _rotate(q.view(-1, heads, head_dim), positions, head_dim, freq)
        k = _rotate(k.view(-1, kv_heads, head_dim), positions, head_dim, freq)
        v = v.view(-1, kv_heads, head_dim)
        mixed, row = torch.empty_like(q), 0
        for r, (first, tokens) in enumerate(sequences):
            rows = slice(row, row + len(tokens))
            keys, values = k[rows], v[rows]
            if first:
                old = [t[n].transpose(0, 1).to(torch.float64) for t in held[r]]
                keys, values = torch.cat([old[0], keys]), torch.cat([old[1], values])
            mixed[rows] = _attend(q[rows], keys, values, head_dim ** -0.5, first)
            row += len(tokens)
        x = x + mixed.reshape(-1, heads * head_dim) @ weights.normal(p + "self_attn.o_proj.weight", (width, heads * head_dim), 0.02).T
        h = _unit(x, eps) * weights.uniform(p + "post_attention_layernorm.weight", (width,), 0.9, 1.1)
        h = (_silu(h @ weights.normal(p + "mlp.gate_proj.weight", (inner, width), 0.02).T)
             * (h @ weights.normal(p + "mlp.up_proj.weight", (inner, width), 0.02).T))
        x = x + h @ weights.normal(p + "mlp.down_proj.weight", (width, inner), 0.02).T
    h = _unit(x[wanted], eps) * weights.uniform("model.norm.weight", (width,), 0.9, 1.1)
    return h @ weights.normal("model.embed_tokens.weight" if tied else "lm_head.weight", (vocab, width), 0.02).T


def _decayed(q, k, v, decay):
    """[T, H, *]: S_t = c S_(t-1) + k_t v_t^T, o_t = S_t^T q_t, written as a sum over earlier tokens."""
    at = torch.arange(q.shape[0], device="cuda", dtype=torch.float64)
    gap = at[:, None] - at[None, :]
    out = []
    for h, c in enumerate(decay):
        factor = torch.where(gap >= 0, c ** gap.clamp(min=0), 0.0)
        out.append(((q[:, h] @ k[:, h].T) * factor) @ v[:, h])
    return torch.stack(out, dim=1)


def mozepel_logits(case, weights, tokens):
    """Logits of the last token of one prompt."""
    width, _heads, _kv, _dim, inner, vocab = SHAPES[case["shape"]][:6]
    config, T = config_of(case), len(tokens)
    eps, alpha = config["norm"]["eps"], config["postln_alpha"]
    at = torch.arange(T, device="cuda")
    x = weights.normal("embed", (vocab, width), 1.0)[torch.tensor(tokens, device="cuda")]
    matrix = lambda name, out, inp: weights.normal(name, (out, inp), inp ** -0.5).T
    norm = lambda name, n: weights.uniform(name, (n,), 0.9, 1.1)

    def retention(p, m):
        H, d = m["heads"], m["dim"]
        q, k, v, gate = (x @ matrix(p + t, H * d, width) for t in ("q", "k", "v", "g"))
        freq = _frequencies(d, m["rot"]["base"])
        q, k = (_rotate(t.view(T, H, d), at, d, freq) for t in (q, k))
        o = _unit(_decayed(q, k * d ** -0.5, v.view(T, H, d), m["decay"]), eps).reshape(T, H * d)
        return (o * _silu(gate)) @ matrix(p + "o", width, H * d)

    def left(p, m):
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        parts = []
        for t, rows in (("q", H), ("k", G), ("v", G)):
            u = x @ matrix(p + t, rows * d, width)
            taps = weights.uniform(f"{p}{t}.conv", (rows * d, m["conv"]), -0.5, 0.5)
            padded = torch.cat([torch.zeros((m["conv"] - 1, rows * d), dtype=u.dtype, device="cuda"), u])
            parts.append(sum(padded[j:j + T] * taps[:, j] for j in range(m["conv"])).view(T, rows, d))
        q, k = (_unit(t, eps) * norm(f"{p}{name}.norm", d) for t, name in zip(parts, "qk"))
        v = parts[2]
        rot = m["rot"]
        freq = _frequencies(rot["dims"], rot["base"], rot["scaling"])
        q, k = (_rotate(t, at, rot["dims"], freq) for t in (q, k))
        size, pool = m["mask"]["size"], m["mask"]["pool"]
        blocks = T // pool
        pooled = [t[:blocks * pool].view(blocks, pool, G, d).mean(1) for t in (k, v)]
        k, v = (torch.cat([a, b]).transpose(0, 1).repeat_interleave(H // G, dim=0) for a, b in zip(pooled, (k, v)))
        ends = torch.arange(1, blocks + 1, device="cuda") * pool - 1
        gap = at[:, None] - at[None, :]
        hidden = torch.cat([ends[None, :] > at[:, None] - size, (gap < 0) | (gap >= size)], dim=1)
        scores = (m["scale"] * (q.transpose(0, 1) @ k.transpose(1, 2))).masked_fill_(hidden, -math.inf)
        return (torch.softmax(scores, dim=-1) @ v).transpose(0, 1).reshape(T, H * d) @ matrix(p + "o", width, H * d)

    def right(p, m):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(x @ matrix(p + t, H * n, width)).view(T, H, n) for t, n in (("q", d), ("k", d), ("v", dv)))
        o = _unit(_decayed(q, k, v, m["decay"]).reshape(T, H * dv), eps) * norm(p + "norm", H * dv)
        return (o * torch.sigmoid(x @ matrix(p + "g", H * dv, width))) @ matrix(p + "o", width, H * dv)

    for n, layer in enumerate(config["layers"]):
        p, m = f"l{n}.", layer["mixer"]
        if layer["type"] == "retention":
            y = retention(p + "mix.", m)
        else:
            y = m["left_scale"] * left(p + "mix.left.", m["left"]) + m["right_scale"] * right(p + "mix.right.", m["right"])
        x = _unit(alpha * x + y, eps) * norm(p + "norm1", width)
        y = (_silu(x @ matrix(p + "mlp.gate", inner, width)) * (x @ matrix(p + "mlp.up", inner, width))) @ matrix(p + "mlp.down", width, inner)
        x = _unit(alpha * x + y, eps) * norm(p + "norm2", width)
    return (_unit(x[-1:], eps) * norm("final.norm", width)) @ matrix("head", vocab, width)


@torch.no_grad()
def exact(case, seed):
    tokens, weights, kind = case_tokens(case, seed), Weights(case, seed), case["kind"]
    if case["design"] == "mozepel":
        return [mozepel_logits(case, weights, tokens[0])]
    if kind == "generate":
        out = []
        for prompt in tokens:
            ids = list(prompt)
            for _ in range(case["new"]):
                ids.append(int(qwen2_logits(case, weights, [(0, ids)], [-1]).argmax()))
            out.append(ids[len(prompt):])
        return np.array(out)
    if kind == "decode":
        sequences = [(length, t) for length, t in zip(held_lengths(case, seed), tokens)]
        return qwen2_logits(case, weights, sequences, list(range(1, 2 * len(tokens), 2)),
                            lambda r, length: held_entries(case, seed, r, length))
    if kind == "mixed":
        sequences = [(length, t) for length, t in zip(held_lengths(case, seed), tokens)] + [(0, tokens[-1])]
        wanted = list(range(case["batch"])) + [case["batch"] + case["tokens"] - 1]
        return qwen2_logits(case, weights, sequences, wanted, lambda r, length: held_entries(case, seed, r, length))
    first = np.cumsum([0] + [len(t) for t in tokens])
    every = lambda places: qwen2_logits(case, weights, [(0, t) for t in tokens], places)
    if kind != "replay":
        return [every([int(end) - 1 for end in first[1:]])]
    done, places = [0] * len(tokens), []
    for step in replay_steps(case, tokens):
        places.append([int(first[r]) + done[r] + place for r, _part, want in step for place in want])
        for r, part, _want in step:
            done[r] += len(part)
    logits = every([place for step in places for place in step])
    ends = np.cumsum([len(step) for step in places])
    return [logits[end - len(step):end] for end, step in zip(ends, places) if step]
