"""What this engine is timed on: steps and short generations of seeded random models through ``ModelRunner``.

A case is one of four kinds of pass:

* ``decode``: one step in which every running request brings one token, after contexts that ``prepare`` has cached.
* ``prefill``: one step with a portion of one prompt, after ``context`` cached tokens (0: a new request, admitted and
  released in the pass).  ``want`` says whose logits are asked for: the last token's (serving) or every token's (scoring).
* ``mixed``: one step with a portion of one prompt beside the single tokens of running requests, as the scheduler makes it.
* ``generate``: requests are admitted, their prompts run in one step, then ``new`` steps of single tokens, then they are
  released.  Single tokens are given and not sampled, so that a rounding cannot send two runs different ways; with
  ``sample`` every step's logits go through the sampler too.

A ``decode``, ``mixed`` or continued ``prefill`` pass sets its requests back to their contexts when it has been enqueued
(``CacheManager.commit``), as a caller that tries another continuation does; every pass then does the same work.

Models: the layer sizes of the Qwen2 family (7B, 1.5B, 0.5B, their full depths) and two of the engine's other designs at
the sizes that ``bench.py --design`` serves, with dense feed-forwards: Geponex (latent attention and lightning attention)
and Sisetar (gated linear attention, attention on chunks beside the delta rule).  Routed experts are left out: which
experts a token takes turns on a rounding, and outputs of two right programs could not be compared.
"""
import hashlib
import math
import random

import torch

PAGE = 64
DEVICE = "cuda:0"
BF16 = "bfloat16"

QWEN2 = {
    "7B": dict(vocab_size=152064, hidden_size=3584, intermediate_size=18944, num_hidden_layers=28, num_attention_heads=28,
               num_key_value_heads=4, head_dim=128, tie_word_embeddings=False),
    "1.5B": dict(vocab_size=151936, hidden_size=1536, intermediate_size=8960, num_hidden_layers=28, num_attention_heads=12,
                 num_key_value_heads=2, head_dim=128, tie_word_embeddings=True),
    "0.5B": dict(vocab_size=151936, hidden_size=896, intermediate_size=4864, num_hidden_layers=24, num_attention_heads=14,
                 num_key_value_heads=2, head_dim=64, tie_word_embeddings=True),
}
# width, feed-forward, recurrent heads with their key and value sizes, attention heads, kv heads and head size, delta-rule
# heads and size, chunk of the attention's mask
DESIGN = {
    "w1024": (1024, 4096, (8, 64, 128), (16, 2, 64), (8, 64), 1024),
    "w4096": (4096, 14336, (16, 128, 256), (32, 8, 128), (16, 128), 2048),
}
DESIGN_VOCAB = 32768
EPS = 1e-6


def listed():
    return [
        # one user of a small model waits for the next token: the smallest decode step, all latency
        {"name": "decode_small_one", "kind": "decode", "model": "0.5B", "dtype": BF16, "batch": 1, "shortest": 700, "longest": 700},
        # the engine's headline workload: eight requests after 1,024-token prompts
        {"name": "decode_7b_eight", "kind": "decode", "model": "7B", "dtype": BF16, "batch": 8, "shortest": 1040, "longest": 1040},
        # a busy server: requests of very different lengths
        {"name": "decode_ragged", "kind": "decode", "model": "1.5B", "dtype": BF16, "batch": 32, "shortest": 64, "longest": 4096},
        # the widest decode batch that the engine captures
        {"name": "decode_wide", "kind": "decode", "model": "0.5B", "dtype": BF16, "batch": 256, "shortest": 512, "longest": 512},
        # scoring of a short text: every token's logits, an odd length
        {"name": "score_short", "kind": "prefill", "model": "0.5B", "dtype": BF16, "tokens": 37, "context": 0, "want": "all"},
        # the prefill of the headline workload
        {"name": "prefill_7b", "kind": "prefill", "model": "7B", "dtype": BF16, "tokens": 2048, "context": 0, "want": "last"},
        # a long document read in portions: one of the last portions
        {"name": "portion_far", "kind": "prefill", "model": "0.5B", "dtype": BF16, "tokens": 2048, "context": 30720, "want": "last"},
        # a step of the scheduler while a prompt comes in: a ragged portion beside decoding requests
        {"name": "mixed_step", "kind": "mixed", "model": "1.5B", "dtype": BF16, "tokens": 611, "context": 1024, "batch": 31,
         "shortest": 64, "longest": 2048},
        # the 32-bit path: a few requests from prompt to sampled tokens
        {"name": "generate_fp32", "kind": "generate", "model": "0.5B", "dtype": "float32", "batch": 3, "shortest": 61, "longest": 233,
         "new": 8, "sample": True},
        # latent and lightning attention: a long prompt
        {"name": "latent_prefill", "kind": "prefill", "model": "geponex w4096", "dtype": BF16, "tokens": 4096, "context": 0, "want": "last"},
        # the same layers from short prompts on, decoding
        {"name": "latent_generate", "kind": "generate", "model": "geponex w1024", "dtype": BF16, "batch": 8, "shortest": 40, "longest": 300,
         "new": 24, "sample": False},
        # recurrences with gates and chunked attention: prompts and decoding
        {"name": "recurrent_generate", "kind": "generate", "model": "sisetar w1024", "dtype": BF16, "batch": 4, "shortest": 200,
         "longest": 1500, "new": 24, "sample": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "mixed", "fp32", "latent", "latent", "recurrent"])
    if kind == "decode":
        model = rng.choice(["7B", "1.5B", "0.5B"])
        batch = _log_int(rng, 1, {"7B": 64, "1.5B": 128, "0.5B": 256}[model])
        longest = min(_log_int(rng, 64, 8192), 131072 // batch, (1 << 16) // batch if model == "7B" else 1 << 20)
        return {"kind": "decode", "model": model, "dtype": BF16, "batch": batch, "shortest": max(16, _log_int(rng, 16, longest)),
                "longest": longest}
    if kind == "prefill":
        model = rng.choice(["7B", "1.5B", "0.5B"])
        tokens = _log_int(rng, 9, 2048)
        context = rng.choice([0, _log_int(rng, 64, 2048 if model == "7B" else 30720)])
        return {"kind": "prefill", "model": model, "dtype": BF16, "tokens": tokens, "context": context,
                "want": "all" if tokens <= 512 and rng.random() < 0.3 else "last"}
    if kind == "mixed":
        return {"kind": "mixed", "model": rng.choice(["1.5B", "0.5B"]), "dtype": BF16, "tokens": _log_int(rng, 17, 2048),
                "context": rng.choice([0, rng.randint(64, 2048)]), "batch": rng.randint(2, 63), "shortest": 64, "longest": _log_int(rng, 128, 2048)}
    if kind == "fp32":
        shortest = _log_int(rng, 8, 256)
        return {"kind": "generate", "model": "0.5B", "dtype": "float32", "batch": rng.randint(1, 4), "shortest": shortest,
                "longest": shortest + rng.randint(0, 256), "new": rng.randint(4, 12), "sample": True}
    size = rng.choice(["w1024", "w4096"])
    if kind == "latent":
        if rng.random() < 0.5:
            return {"kind": "prefill", "model": "geponex " + size, "dtype": BF16, "tokens": _log_int(rng, 24, 4096), "context": 0, "want": "last"}
        shortest = _log_int(rng, 16, 512)
        return {"kind": "generate", "model": "geponex " + size, "dtype": BF16, "batch": _log_int(rng, 1, 12), "shortest": shortest,
                "longest": shortest + rng.randint(0, 256), "new": rng.randint(8, 24), "sample": False}
    shortest = _log_int(rng, 16, 700)
    return {"kind": "generate", "model": "sisetar " + size, "dtype": BF16, "batch": rng.randint(1, 8), "shortest": shortest,
            "longest": shortest + rng.randint(0, 700), "new": rng.randint(8, 24), "sample": False}


# ---- models: their configurations and seeded random weights ----------------------------------------------------------


def _config(case):
    """The model's config.json."""
    name = case["model"]
    if name in QWEN2:
        return dict(QWEN2[name], architectures=["Qwen2ForCausalLM"], rms_norm_eps=EPS, rope_theta=1e6, max_position_embeddings=32768,
                    use_sliding_window=False, torch_dtype=case["dtype"])
    design, size = name.split()
    width, ff, rec, att, delta, chunk = DESIGN[size]
    heads, kv_heads, dim = att
    layers = []
    for i in range(2):
        if design == "geponex":
            rot = {"dims": dim // 2, "base": 1e6}
            if i == 0:
                rot["scaling"] = {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}
            layers.append({"type": "latent_attention_2" if i else "latent_attention", "mlp": {"kind": "dense", "ff": ff}, "mixer": {
                "heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "q_rank": 12 * dim, "kv_rank": 4 * dim,
                "scale": (1.5 * dim) ** -0.5, "rot": rot}})
            layers.append({"type": "lightning", "mlp": {"kind": "dense", "ff": ff}, "mixer": {
                "heads": rec[0], "dim": rec[1], "vdim": rec[2], "decay": [1.0 - 2.0 ** (-5 - 0.5 * h) for h in range(rec[0])]}})
        else:
            layers.append({"type": "gla", "mixer": {"heads": rec[0], "dim": rec[1], "vdim": rec[2], "tau": 16.0}, "mlp": None})
            layers.append({"type": "parallel", "mlp": {"kind": "dense", "ff": ff}, "mixer": {
                "left": {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "rot": {"dims": dim // 2, "base": 1e6},
                         "scale": dim ** -0.5, "mask": {"size": chunk}},
                "right": {"heads": delta[0], "dim": delta[1]}, "left_scale": 1.0, "right_scale": 1.0}})
    if design == "geponex":
        return {"architecture": "Geponex", "vocab": DESIGN_VOCAB, "width": width, "layers": layers, "norm": {"eps": EPS, "groups": 2},
                "postln_alpha": 2.0}
    return {"architecture": "Sisetar", "vocab": DESIGN_VOCAB, "width": width, "layers": layers, "embedding": {"scale": 1.0},
            "logit_scale": 1.0, "logit_softcap": 30.0, "norm": {"eps": EPS}}


def _generator(seed, name, device=DEVICE):
    g = torch.Generator(device=device)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    return g


def _weight(name, shape, seed, dtype):
    """Tensor ``name`` of the model of this seed, as a checkpoint stores it.  Matrices give outputs of unit size for inputs of
    unit size; queries and keys are larger, so that attention picks some of its keys; what a sublayer adds to the stream
    is a part of what stands there."""
    g = _generator(seed, name)
    r = torch.randn(tuple(shape), generator=g, device=DEVICE, dtype=dtype)
    last = name.split(".")[-2 if name.endswith((".weight", ".bias")) else -1]
    if last == "shift":
        return torch.rand(tuple(shape), generator=g, device=DEVICE, dtype=torch.float32).to(dtype)
    if last == "act":
        return (r * 0.1 + 0.5).to(dtype)
    if "norm" in last:
        return r.mul_(0.1).add_(1.0)
    if len(shape) == 1:
        return r.mul_(0.1)
    if last in ("embed_tokens", "embed", "lm_head"):
        return r.mul_(2.0 * shape[1] ** -0.5)
    gain = {"q_proj": 1.5, "k_proj": 1.5, "uq": 1.5, "uk": 1.5}.get(last, 1.0)
    if last in ("o_proj", "down_proj"):         # the stream of these models is as large as the embedding's rows
        gain = 1.5 * shape[0] ** -0.5
    return r.mul_(gain * shape[1] ** -0.5)


def _runner(case, seed, tokens, requests, longest):
    from vt_transformer_b200 import ModelRunner
    from vt_transformer_b200.config import config_from_dict
    from vt_transformer_b200.weights import DictSource
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16

    def source(table):
        return DictSource({n: _weight(n, s.made_shape(), seed, dtype) for n, s in table.items() if not s.optional})
    return ModelRunner.build(config_from_dict(_config(case)), source, dtype=case["dtype"], device=DEVICE, page_size=PAGE,
                             num_pages=tokens // PAGE + 2 * requests + 2, max_requests=requests, max_seq_len=longest)


# ---- inputs ---------------------------------------------------------------------------------------------------------------


def _lengths(case, seed):
    """The requests' cached lengths (or prompts), spread over the logarithm between the two ends; the longest is there."""
    rng = random.Random(f"{seed}:lengths")
    lo, hi = min(case["shortest"], case["longest"]), case["longest"]
    got = [_log_int(rng, lo, hi) for _ in range(case["batch"])]
    got[rng.randrange(len(got))] = hi
    return got


def _tokens(case, seed, count, what):
    vocab = QWEN2[case["model"]]["vocab_size"] if case["model"] in QWEN2 else DESIGN_VOCAB
    g = torch.Generator().manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{what}".encode()).digest()[:7], "little"))
    return torch.randint(0, vocab, (count,), generator=g).tolist()


def _requests(case, seed):
    """A request each: (its cached tokens, the tokens that the pass brings)."""
    kind = case["kind"]
    if kind == "prefill":
        return [(_tokens(case, seed, case["context"], "context"), _tokens(case, seed, case["tokens"], "portion"))]
    if kind == "generate":
        return [([], _tokens(case, seed, n + case["new"], f"request {i}")) for i, n in enumerate(_lengths(case, seed))]
    out = [(_tokens(case, seed, n, f"request {i}"), _tokens(case, seed, 1, f"token {i}")) for i, n in enumerate(_lengths(case, seed))]
    if kind == "mixed":
        out.append((_tokens(case, seed, case["context"], "context"), _tokens(case, seed, case["tokens"], "portion")))
    return out


def prepare(case, seed):
    from vt_transformer_b200 import SamplingParams, StepEntry
    requests = _requests(case, seed)
    longest = -(-max(len(c) + len(t) for c, t in requests) // PAGE) * PAGE
    runner = _runner(case, seed, sum(len(c) + len(t) for c, t in requests), len(requests), longest)
    state = {"case": case, "runner": runner, "entry": StepEntry, "requests": [t for _, t in requests]}
    if case["kind"] == "generate":
        state["new"] = case["new"]
        if case.get("sample"):
            from vt_transformer_b200.sampling import Sampler
            state["sampler"] = Sampler(runner.rt.ops, runner.rt.device)
            kinds = [SamplingParams(temperature=0.0), SamplingParams(temperature=0.8, top_p=0.95), SamplingParams(temperature=1.0, top_k=50),
                     SamplingParams(temperature=0.7, top_k=40, top_p=0.9)]
            state["params"] = [kinds[(seed + i) % 4] for i in range(len(requests))]
        return state
    if case["kind"] == "prefill" and not requests[0][0]:
        return state
    # the contexts, in portions of up to 4,096 tokens a step
    rows = [runner.admit() for _ in requests]
    for row, (context, _) in zip(rows, requests):
        for a in range(0, len(context), 4096):
            runner.step([StepEntry(row, context[a:a + 4096], [])])
    state["rows"] = rows
    state["lengths"] = [len(c) for c, _ in requests]
    return state


# ---- the pass -----------------------------------------------------------------------------------------------------------------


def run(state):
    case, runner, Entry, requests = state["case"], state["runner"], state["entry"], state["requests"]
    if case["kind"] == "generate":
        return _generate(state)
    rows = state.get("rows") or [runner.admit()]
    entries = []
    for row, tokens in zip(rows, requests):
        every = case.get("want") == "all"
        entries.append(Entry(row, tokens, list(range(len(tokens))) if every else [len(tokens) - 1]))
    logits = runner.step(entries)
    if "rows" in state:
        for row, n in zip(rows, state["lengths"]):
            runner.cache.commit(row, n)
    else:
        runner.release(rows[0])
    return logits


def _generate(state):
    runner, Entry, requests, new = state["runner"], state["entry"], state["requests"], state["new"]
    rows = [runner.admit() for _ in requests]
    out, picked = [], []
    for i in range(new + 1):
        if i == 0:
            entries = [Entry(row, t[:len(t) - new], [len(t) - new - 1]) for row, t in zip(rows, requests)]
        else:
            entries = [Entry(row, [t[len(t) - new + i - 1]], [0]) for row, t in zip(rows, requests)]
        logits = runner.step(entries)
        if "sampler" in state:
            picked.append(state["sampler"].sample(logits, state["params"], [i] * len(rows)))
        out.append(logits.clone())          # a captured step's logits are overwritten by the next
    for row in rows:
        runner.release(row)
    return {"logits": out, "picked": picked}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------


def _sizes(case):
    """(weights that every step multiplies with, values of the head, values cached a token that all later tokens read,
    attention flops a (token, key), recurrent state values a request)."""
    name = case["model"]
    if name in QWEN2:
        c = QWEN2[name]
        H, kv = c["hidden_size"], c["num_key_value_heads"] * c["head_dim"]
        layer = H * (2 * H + 2 * kv) + 3 * H * c["intermediate_size"]
        n = c["num_hidden_layers"]
        return n * layer, H * c["vocab_size"], n * 2 * kv, n * 4 * H, 0
    design, size = name.split()
    W, ff, rec, att, delta, chunk = DESIGN[size]
    heads, kv_heads, dim = att
    state = rec[0] * rec[1] * rec[2]
    if design == "geponex":
        q_rank, kv_rank, r = 12 * dim, 4 * dim, dim // 2
        attn = W * q_rank + q_rank * heads * (dim + r) + W * (kv_rank + r) + 2 * heads * dim * kv_rank + heads * dim * W
        light = W * (2 * rec[0] * rec[1] + 2 * rec[0] * rec[2]) + rec[0] * rec[2] * W
        return (2 * (attn + light) + heads * dim * W + 4 * 2 * W * ff, W * DESIGN_VOCAB, 2 * (kv_rank + r),
                2 * 2 * heads * (2 * dim + r), 2 * state)
    gla = W * (2 * rec[0] * rec[1] + 2 * rec[0] * rec[2] + 16) + 16 * rec[0] * rec[1] + rec[0] * rec[2] * W
    d = delta[0] * delta[1]
    par = W * (heads * dim + 2 * kv_heads * dim) + heads * dim * W + 5 * W * d + 16 * (W + d) + d * W
    return (2 * (gla + par) + 2 * 2 * W * ff, W * DESIGN_VOCAB, 2 * 2 * kv_heads * dim, 2 * 4 * heads * dim,
            2 * (state + delta[0] * delta[1] * delta[1]))


def work(case):
    """Weights once a step, cached values once a step for every request (a chunk's attention sees what its chunk holds),
    states read and written once a step, logits once; the products' and the attention's multiply-adds."""
    weights, head, cached, att, state = _sizes(case)
    item = 4 if case["dtype"] == "float32" else 2
    requests = _requests(dict(case), 0)
    vocab = QWEN2[case["model"]]["vocab_size"] if case["model"] in QWEN2 else DESIGN_VOCAB
    reach = DESIGN[case["model"].split()[1]][5] if case["model"].startswith("sisetar") else 1 << 40
    steps = []                                   # a step: [(cached before, tokens, logits wanted)]
    if case["kind"] == "generate":
        new = case["new"]
        steps.append([(0, len(t) - new, 1) for _, t in requests])
        steps += [[(len(t) - new + i, 1, 1) for _, t in requests] for i in range(new)]
    else:
        steps.append([(len(c), len(t), len(t) if case.get("want") == "all" else 1) for c, t in requests])
    total_bytes = total_flops = 0
    for step in steps:
        total_bytes += (weights + head) * item
        for before, n, wanted in step:
            seen = sum(min(p % reach, p) + 1 for p in range(before, before + n)) if reach < 1 << 40 else n * before + n * (n + 1) // 2
            total_bytes += (before % reach + n) * cached * item + 2 * 4 * state + wanted * vocab * 4
            total_flops += 2 * weights * n + 2 * head * wanted + att * seen + 4 * state * n
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3, "differ": 0.01}
    return {"rel": 0.03, "max": 0.5}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------

F = torch.float64


def _rms(x, w=None, groups=1):
    y = x.reshape(*x.shape[:-1], groups, -1)
    y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + EPS)).reshape(x.shape)
    return y if w is None else y * w


def _causal(q, k, v, first, scale, sink=None, chunk=None):
    """q [T, H, d], its token t at position first + t; k [S, G, d], v [S, G, e] at positions 0..S-1; heads in groups."""
    T, H, _ = q.shape
    S, G, _ = k.shape
    out = torch.empty(T, H, v.shape[2], dtype=F, device=q.device)
    kk, vv = k.permute(1, 2, 0), v.permute(1, 0, 2)
    block = max(1, min(T, (1 << 27) // (S * H)))
    for a in range(0, T, block):
        b = min(T, a + block)
        n = min(S, first + b)
        qq = q[a:b].reshape(b - a, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, -1, q.shape[2])
        s = (torch.bmm(qq, kk[:, :, :n]) * scale).reshape(G, H // G, b - a, n)
        pos, key = torch.arange(first + a, first + b, device=q.device)[:, None], torch.arange(n, device=q.device)[None]
        hidden = key > pos
        if chunk:
            hidden |= torch.div(key, chunk, rounding_mode="floor") != torch.div(pos, chunk, rounding_mode="floor")
        s.masked_fill_(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.reshape(G, H // G, 1, 1).expand(-1, -1, b - a, 1)], dim=3)
        p = torch.softmax(s, dim=-1)[..., :n]
        out[a:b] = torch.bmm(p.reshape(G, -1, n), vv[:, :n]).reshape(G, H // G, b - a, -1).permute(2, 0, 1, 3).reshape(b - a, H, -1)
    return out


def _turn(x, first, dims, base, interleaved=False, ramp=None):
    """x [T, heads, d] at positions first..: the first ``dims`` dimensions of a head in pairs (i, i + dims / 2), or side by side."""
    half = dims // 2
    i = torch.arange(half, dtype=F, device=x.device)
    freq, mult = base ** (-2.0 * i / dims), 1.0
    if ramp:
        pair = lambda turns: dims * math.log(ramp["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(pair(ramp["fast"])), 0), min(math.ceil(pair(ramp["slow"])), dims - 1)
        part = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        freq, mult = freq / ramp["factor"] * part + freq * (1 - part), 0.1 * math.log(ramp["factor"]) + 1.0
    ang = torch.arange(first, first + x.shape[0], dtype=F, device=x.device)[:, None] * freq[None]
    c, s = (torch.cos(ang) * mult)[:, None], (torch.sin(ang) * mult)[:, None]
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, half), slice(half, dims))
    u, v = x[..., a], x[..., b]
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def _exact_qwen2(c, get, seqs, wanted):
    H, n, g, d = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    embed = get("model.embed_tokens.weight", (c["vocab_size"], H), keep=True)
    x = embed[torch.as_tensor([t for s in seqs for t in s], device=DEVICE)].to(F)
    ends = [0]
    for s in seqs:
        ends.append(ends[-1] + len(s))
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        lin = lambda y, name, rows: y @ get(f"{p}self_attn.{name}.weight", (rows, H)).T + get(f"{p}self_attn.{name}.bias", (rows,))
        h = _rms(x, get(p + "input_layernorm.weight", (H,)))
        q, k, v = (lin(h, name, rows * d).reshape(-1, rows, d) for name, rows in (("q_proj", n), ("k_proj", g), ("v_proj", g)))
        o = torch.cat([_causal(_turn(q[a:b], 0, d, 1e6), _turn(k[a:b], 0, d, 1e6), v[a:b], 0, d ** -0.5) for a, b in zip(ends, ends[1:])])
        x = x + o.reshape(-1, n * d) @ get(p + "self_attn.o_proj.weight", (H, n * d)).T
        h = _rms(x, get(p + "post_attention_layernorm.weight", (H,)))
        ff = c["intermediate_size"]
        gate, up, down = (get(f"{p}mlp.{m}_proj.weight", (H, ff) if m == "down" else (ff, H)) for m in ("gate", "up", "down"))
        for a in range(0, x.shape[0], 16384):
            x[a:a + 16384] += (torch.nn.functional.silu(h[a:a + 16384] @ gate.T) * (h[a:a + 16384] @ up.T)) @ down.T
    rows = torch.cat([x[a:b][torch.as_tensor(w, device=DEVICE)] for a, b, w in zip(ends, ends[1:], wanted)])
    head = embed.to(F) if c["tie_word_embeddings"] else get("lm_head.weight", (c["vocab_size"], H))
    return _rms(rows, get("model.norm.weight", (H,))) @ head.T


def _exact_geponex(c, get, seqs, wanted):
    W, silu = c["width"], torch.nn.functional.silu
    embed, out = get("embed", (c["vocab"], W)), []
    for ids, want in zip(seqs, wanted):
        x = embed[torch.as_tensor(ids, device=DEVICE)]
        T = x.shape[0]
        for i, layer in enumerate(c["layers"]):
            m, p = layer["mixer"], f"l{i}."
            lin = lambda y, name, rows: y @ get(f"{p}mix.{name}", (rows, y.shape[1])).T
            h = x + (torch.cat([torch.zeros_like(x[:1]), x[:-1]]) - x) * get(p + "shift", (W,))
            if layer["type"] == "lightning":
                n, d, e = m["heads"], m["dim"], m["vdim"]
                q, k, v = (silu(lin(h, name, n * z)).reshape(T, n, z).transpose(0, 1) for name, z in (("q", d), ("k", d), ("v", e)))
                S = torch.zeros(n, d, e, dtype=F, device=DEVICE)
                decay = torch.tensor(m["decay"], dtype=F, device=DEVICE)[:, None]
                pieces = []
                for a in range(0, T, 256):          # the state carried over runs of 256 tokens, their own terms as a product
                    b = min(T, a + 256)
                    t = torch.arange(b - a, dtype=F, device=DEVICE)
                    gap = t[:, None] - t[None, :]
                    inner = torch.bmm(q[:, a:b], k[:, a:b].transpose(1, 2)) * torch.where(gap >= 0, decay[:, :, None] ** gap.clamp(min=0), 0)
                    pieces.append(torch.bmm(inner, v[:, a:b]) + torch.bmm(q[:, a:b] * (decay ** (t + 1))[:, :, None], S))
                    S = S * (decay ** (b - a))[:, :, None] + torch.bmm((k[:, a:b] * (decay ** (b - a - 1 - t))[:, :, None]).transpose(1, 2), v[:, a:b])
                o = torch.cat(pieces, dim=1).transpose(0, 1).reshape(T, n * e)
                y = lin(_rms(o, get(p + "mix.norm", (n * e,))) * torch.sigmoid(lin(h, "g", n * e)), "o", W)
            else:
                n, d, r, e, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
                turn = lambda z: _turn(z, 0, m["rot"]["dims"], m["rot"]["base"], True, m["rot"].get("scaling"))
                q = lin(_rms(lin(h, "dq", m["q_rank"]), get(p + "mix.dq.norm", (m["q_rank"],))), "uq", n * (d + r)).reshape(T, n, d + r)
                down = lin(h, "dkv", rank + r)
                latent = _rms(down[:, :rank], get(p + "mix.dkv.norm", (rank,)))
                k = torch.cat([lin(latent, "uk", n * d).reshape(T, n, d), turn(down[:, None, rank:]).expand(-1, n, -1)], dim=-1)
                second = layer["type"] == "latent_attention_2"
                o = _causal(torch.cat([q[..., :d], turn(q[..., d:])], dim=-1), k, lin(latent, "uv", n * e).reshape(T, n, e), 0, m["scale"],
                            get(p + "mix.sink", (n,)) if second else None).reshape(T, n * e)
                if second:
                    o = o * torch.sigmoid(lin(h, "g", n * e))
                y = lin(o, "o", W)
            x = _rms(c["postln_alpha"] * x + y, get(p + "norm1", (W,)), c["norm"]["groups"])
            ff, p = layer["mlp"]["ff"], p + "mlp."
            z = x @ get(p + "up", (ff, W)).T + get(p + "up.b", (ff,))
            act = torch.nn.functional.softplus(get(p + "act", (2,)))
            z = torch.where(z > 0, act[0] * z * z, (0.5 + act[1]) * (torch.expm1(z.clamp(max=0)) - z)) + z / 2
            x = _rms(c["postln_alpha"] * x + z @ get(p + "down", (W, ff)).T + get(p + "down.b", (W,)), get(f"l{i}.norm2", (W,)), c["norm"]["groups"])
        out.append(_rms(x[torch.as_tensor(want, device=DEVICE)], get("final.norm", (W,)), c["norm"]["groups"]) @ embed.T)
    return torch.cat(out)


def _layer_norm(x, w):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _exact_sisetar(c, get, seqs, wanted):
    """All sequences side by side, padded at their ends (no token sees a later one)."""
    W, B, T = c["width"], len(seqs), max(len(s) for s in seqs)
    ids = torch.zeros(B, T, dtype=torch.long, device=DEVICE)
    for b, s in enumerate(seqs):
        ids[b, :len(s)] = torch.as_tensor(s, device=DEVICE)
    embed = get("embed", (c["vocab"], W))
    x = embed[ids]
    for i, layer in enumerate(c["layers"]):
        p = f"l{i}."
        lin = lambda y, name, rows: y @ get(f"{p}mix.{name}", (rows, y.shape[-1])).T
        h = _layer_norm(x, get(p + "norm1", (W,)))
        if layer["type"] == "gla":
            m = layer["mixer"]
            n, d, e = m["heads"], m["dim"], m["vdim"]
            q, k, v = (lin(h, name, n * z).reshape(B, T, n, z) for name, z in (("q", d), ("k", d), ("v", e)))
            alpha = torch.sigmoid(lin(lin(h, "a1", 16), "a2", n * d) + get(p + "mix.a2.b", (n * d,))) ** (1.0 / m["tau"])
            alpha = alpha.reshape(B, T, n, d, 1)
            S, o = torch.zeros(B, n, d, e, dtype=F, device=DEVICE), torch.empty(B, T, n, e, dtype=F, device=DEVICE)
            for t in range(T):
                S = S.mul_(alpha[:, t]).add_(k[:, t, :, :, None] * v[:, t, :, None, :])
                o[:, t] = torch.matmul(q[:, t, :, None, :], S)[..., 0, :]
            o = _rms(o * d ** -0.5) * get(p + "mix.norm", (e,))
            x = x + lin(o.reshape(B, T, n * e) * torch.nn.functional.silu(lin(h, "g", n * e)), "o", W)
            continue
        m = layer["mixer"]["left"]
        n, g, d = m["heads"], m["kv_heads"], m["dim"]
        y = torch.empty(B, T, n * d, dtype=F, device=DEVICE)
        for b in range(B):
            q, k, v = (lin(h[b], "left." + name, z * d).reshape(T, z, d) for name, z in (("q", n), ("k", g), ("v", g)))
            q, k = (_rms(_turn(z, 0, m["rot"]["dims"], m["rot"]["base"])) for z in (q, k))
            y[b] = _causal(q, k, v, 0, m["scale"], chunk=m["mask"]["size"]).reshape(T, n * d)
        left = lin(y, "left.o", W)
        m = layer["mixer"]["right"]
        n, d = m["heads"], m["dim"]
        low = torch.tanh(lin(h, "right.w1", 16)) @ get(p + "mix.right.w2", (n * d, 16)).T + get(p + "mix.right.w0", (n * d,))
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(low)).reshape(B, T, n, d, 1)
        a = torch.sigmoid(lin(h, "right.a", n * d) + get(p + "mix.right.a.b", (n * d,))).reshape(B, T, n, d)
        r, k, v = (lin(h, "right." + name, n * d).reshape(B, T, n, d) for name in ("r", "k", "v"))
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S, o = torch.zeros(B, n, d, d, dtype=F, device=DEVICE), torch.empty(B, T, n, d, dtype=F, device=DEVICE)
        for t in range(T):
            uS = torch.matmul(u[:, t, :, None, :], S)
            S = S * decay[:, t] - (a * u)[:, t, :, :, None] * uS + k[:, t, :, :, None] * v[:, t, :, None, :]
            o[:, t] = torch.matmul(r[:, t, :, None, :], S)[..., 0, :]
        o = _rms(o).reshape(B, T, n * d) * get(p + "mix.right.norm", (n * d,))
        x = x + left + lin(o * torch.sigmoid(lin(h, "right.g", n * d)), "right.o", W)
        h, ff, p = _layer_norm(x, get(p + "norm2", (W,))), layer["mlp"]["ff"], p + "mlp."
        z, act = h @ get(p + "up", (ff, W)).T, get(p + "act", (4,))
        x = x + (act[0] * _rms(z) + act[1] * _rms(z * z) + act[2] * _rms(z * z * z) + act[3]) @ get(p + "down", (W, ff)).T
    rows = torch.cat([x[b][torch.as_tensor(w, device=DEVICE)] for b, w in enumerate(wanted)])
    cap = c["logit_softcap"]
    return cap * torch.tanh(_layer_norm(rows, get("final.norm", (W,))) @ embed.T / cap)


def exact(case, seed):
    config, requests = _config(case), _requests(case, seed)
    stored = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    kept = {}

    def get(name, shape, keep=False):
        """A weight in 64 bits (the largest, with ``keep``, as it is stored)."""
        if keep:
            return _weight(name, shape, seed, stored)
        small = math.prod(shape) <= 1 << 22 or name == "embed"
        if name in kept:
            return kept[name]
        w = _weight(name, shape, seed, stored).to(F)
        if small:
            kept[name] = w
        return w
    seqs, new = [c + t for c, t in requests], case.get("new", 0)
    if case["kind"] == "generate":
        wanted = [list(range(len(s) - new - 1, len(s))) for s in seqs]
    elif case.get("want") == "all":
        wanted = [list(range(len(c), len(c) + len(t))) for c, t in requests]
    else:
        wanted = [[len(s) - 1] for s in seqs]
    fn = {"Geponex": _exact_geponex, "Sisetar": _exact_sisetar}.get(config.get("architecture"), _exact_qwen2)
    logits = fn(config, get, seqs, wanted)
    if case["kind"] != "generate":
        return logits
    by_request = logits.reshape(len(seqs), new + 1, -1)
    return {"logits": [by_request[:, i] for i in range(new + 1)], "picked": [None] * (new + 1) if case.get("sample") else []}
