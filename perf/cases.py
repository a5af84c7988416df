"""The workloads by which the engine's speed is judged: steps of the model over a batch of requests, as the engine, the
benchmark and the trace program make them (`ModelRunner.step`), and short lives of whole requests.

A step takes any mix of single tokens (requests that decode) and prompt portions, so one kind of case covers decoding,
prompts and continuous batching: `decode` requests bring one token each behind a context of `ctx_lo` to `ctx_hi` cached
tokens, `prompts` requests share `prompt_tokens` new tokens behind `prompt_cached` cached ones each.  The logits that the
sampler would be given (one row per request) come back.  A life starts `prompts` requests, runs their prompts in one step and then
`new_tokens` steps of one given token each, all from the cache that the steps before left; every step's logits come back.

Models are the benchmark's: the layer sizes of Llama-3-8B, Llama-3.2-1B and Llama-2-13B with all their layers, and the
Dizepel design at its benchmark's smaller size.  Designs with routed experts are left out: which expert a token goes to is decided
by a comparison, two correct 16-bit implementations decide some tokens differently, and their logits then differ by far
more than rounding.  Weights and cached keys and values are random, drawn by tensor name.
"""
import hashlib
import math
import random

import torch

V_LLAMA3 = 128256
_8B = dict(architectures=["LlamaForCausalLM"], model_type="llama", hidden_size=4096, num_hidden_layers=32,
           num_attention_heads=32, num_key_value_heads=8, head_dim=128, intermediate_size=14336, vocab_size=V_LLAMA3,
           rope_theta=500000.0, rms_norm_eps=1e-5, tie_word_embeddings=False, max_position_embeddings=8192,
           hidden_act="silu", torch_dtype="bfloat16", bos_token_id=128000, eos_token_id=128001)
_1B = dict(_8B, hidden_size=2048, num_hidden_layers=16, head_dim=64, intermediate_size=8192, tie_word_embeddings=True,
           max_position_embeddings=131072,
           rope_scaling=dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0,
                             original_max_position_embeddings=8192))
_13B = dict(_8B, hidden_size=5120, num_hidden_layers=40, num_attention_heads=40, num_key_value_heads=40,
            intermediate_size=13824, vocab_size=32000, rope_theta=10000.0, max_position_embeddings=4096, bos_token_id=1,
            eos_token_id=2)
_PAIR = {"type": "parallel", "mlp": {"kind": "dense", "ff": 4096},
         "mixer": {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "conv": 4, "softcap": 30.0,
                            "rot": {"dims": 64, "base": 5.0e5,
                                    "scaling": {"factor": 16.0, "original": 4096, "fast": 32.0, "slow": 1.0}}},
                   "right": {"heads": 32, "vdim": 64, "state": 128, "groups": 4, "conv": 4, "norm_groups": 4}}}
_DIZEPEL = {"architecture": "Dizepel", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.5},
            "canon": {"taps": 4}, "loop": {"start": 0, "stop": 4, "times": 1}, "layers": [_PAIR] * 4}
MODELS = {"llama3-8b": _8B, "llama3.2-1b": _1B, "llama2-13b": _13B, "dizepel": _DIZEPEL}
MAX_LEN = {"llama3-8b": 8192, "llama3.2-1b": 8192, "llama2-13b": 4096, "dizepel": 8192}
BLOCK = 16            # tokens per cache page
CYCLE = 16            # steps that decoding goes on for before it starts again from the same contexts
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def _step(name, model, decode=0, ctx=(0, 0), prompts=0, prompt_tokens=0, prompt_cached=0, dtype="bfloat16"):
    return dict(name=name, kind="step", model=model, dtype=dtype, decode=decode, ctx_lo=ctx[0], ctx_hi=ctx[1], prompts=prompts,
                prompt_tokens=prompt_tokens, prompt_cached=prompt_cached)


def _life(name, model, prompts, prompt_tokens, new_tokens, dtype="bfloat16"):
    return dict(name=name, kind="life", model=model, dtype=dtype, prompts=prompts, prompt_tokens=prompt_tokens, new_tokens=new_tokens)


def listed():
    return [
        # one user of a small model early in an answer: the least work a step can have
        _step("1b decode 1", "llama3.2-1b", decode=1, ctx=(97, 97)),
        # the benchmark's headline: eight requests of 2,048 tokens
        _step("8b decode 8", "llama3-8b", decode=8, ctx=(2047, 2047)),
        # a server between its busy hours: an odd number of requests at every stage of their answers
        _step("8b decode 27 ragged", "llama3-8b", decode=27, ctx=(130, 2300)),
        # a full batch of a small model, as in the benchmark's serving run
        _step("1b decode 64 ragged", "llama3.2-1b", decode=64, ctx=(130, 2300)),
        # a full batch of long contexts
        _step("8b decode 64", "llama3-8b", decode=64, ctx=(2047, 2047)),
        # heads that are not grouped, near the longest context that the model takes
        _step("13b decode 5", "llama2-13b", decode=5, ctx=(3900, 3900)),
        # a short question to a small model: the time to its first token
        _step("1b prompt 77", "llama3.2-1b", prompts=1, prompt_tokens=77),
        # the benchmark's prompt
        _step("8b prompt 2048", "llama3-8b", prompts=1, prompt_tokens=2048),
        # a full step of the engine's default budget: several documents of unequal length at once
        _step("8b prompts 8192", "llama3-8b", prompts=3, prompt_tokens=8192),
        # continuous batching: a later portion of a long prompt beside requests that decode
        _step("8b mixed", "llama3-8b", decode=63, ctx=(130, 2300), prompts=1, prompt_tokens=1985, prompt_cached=1003),
        # 32-bit throughout, as it is run to check a model: prompts, then tokens one by one
        _life("1b life float32", "llama3.2-1b", prompts=3, prompt_tokens=515, new_tokens=12, dtype="float32"),
        # a design with attention beside a recurrence: prompts, then tokens one by one
        _life("dizepel life", "dizepel", prompts=5, prompt_tokens=3001, new_tokens=24),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "float32", "dizepel"])
    if kind == "decode":
        model = rng.choice(["llama3-8b", "llama3.2-1b", "llama2-13b"])
        most = {"llama3-8b": 2300, "llama3.2-1b": 4000, "llama2-13b": 3900}[model]
        n = _log_int(rng, 1, 8 if model == "llama2-13b" else 64)
        if model == "llama2-13b":
            most = min(most, 5 * 3900 // n)
        hi = _log_int(rng, 32, most)
        c = _step("", model, decode=n, ctx=(rng.choice([hi, max(16, hi // 17)]), hi))
    elif kind == "prompt":
        total = _log_int(rng, 17, 8191)
        c = _step("", rng.choice(["llama3-8b", "llama3.2-1b"]), prompts=rng.choice([1, 1, 2, 3, 4]), prompt_tokens=total,
                  prompt_cached=rng.choice([0, 0, 0, rng.randint(1, 1500)]))
    elif kind == "mixed":
        hi = _log_int(rng, 100, 2300)
        c = _step("", rng.choice(["llama3-8b", "llama3.2-1b"]), decode=_log_int(rng, 1, 63), ctx=(max(16, hi // 17), hi),
                  prompts=rng.choice([1, 2]), prompt_tokens=_log_int(rng, 32, 2000), prompt_cached=rng.choice([0, rng.randint(1, 2000)]))
    elif kind == "float32":
        c = _life("", "llama3.2-1b", prompts=rng.choice([1, 2, 3, 6]), prompt_tokens=_log_int(rng, 24, 600), new_tokens=rng.randint(2, 16),
                  dtype="float32")
    else:
        c = _life("", "dizepel", prompts=rng.randint(1, 12), prompt_tokens=_log_int(rng, 64, 4000), new_tokens=rng.randint(4, 32))
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ sizes of a case

def _split(total, parts):
    """`total` tokens over `parts` prompts of unequal length, each at least one."""
    parts = min(parts, total)
    w = [1.0 / (i + 1) ** 0.7 for i in range(parts)]
    n = [max(1, int(total * x / sum(w))) for x in w]
    n[0] += total - sum(n)
    return n


def _requests(case):
    """[(cached tokens, new tokens)] of a step or of a life's first step."""
    if case["kind"] == "life":
        return [(0, n) for n in _split(case["prompt_tokens"], case["prompts"])]
    rng = random.Random(case["decode"] * 1000003 + case["ctx_hi"])
    lens = [rng.randint(case["ctx_lo"], case["ctx_hi"]) for _ in range(case["decode"])]
    if lens:
        lens[0] = case["ctx_hi"]
    return [(c, 1) for c in lens] + ([(case["prompt_cached"], n) for n in _split(case["prompt_tokens"], case["prompts"])] if case["prompts"] else [])


def _llama_params(m):
    H, I, d = m["hidden_size"], m["intermediate_size"], m["head_dim"]
    q, kv = m["num_attention_heads"] * d, m["num_key_value_heads"] * d
    return m["num_hidden_layers"] * (H * (2 * q + 2 * kv) + 3 * H * I), H * m["vocab_size"]


def _dizepel_params(m):
    D, total = m["width"], 0
    for L in m["layers"]:
        a, b = L["mixer"]["left"], L["mixer"]["right"]
        q, kv, inner = a["heads"] * a["dim"], a["kv_heads"] * a["dim"], b["heads"] * b["vdim"]
        total += D * (2 * q + kv) + D * (3 * inner + 2 * b["groups"] * b["state"] + b["heads"]) + 2 * D * L["mlp"]["ff"]
    return total, D * m["vocab"]


def _step_work(case, requests):
    """Weights read once, cached keys and values read once, new ones written, logits written; the products and the
    attention over the keys that each token sees."""
    m, e = MODELS[case["model"]], 4 if case["dtype"] == "float32" else 2
    T, rows = sum(n for _, n in requests), len(requests)
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in requests)            # (query, key) pairs
    if case["model"] == "dizepel":
        body, head = _dizepel_params(m)
        a, b = m["layers"][0]["mixer"]["left"], m["layers"][0]["mixer"]["right"]
        layers, heads, d, kv = len(m["layers"]), a["heads"], a["dim"], a["kv_heads"] * a["dim"]
        state = b["heads"] * b["vdim"] * b["state"]
        extra_bytes, extra_flops = layers * len(requests) * state * 8, layers * T * state * 5
        width, vocab = m["width"], m["vocab"]
    else:
        body, head = _llama_params(m)
        layers, heads, d, kv = m["num_hidden_layers"], m["num_attention_heads"], m["head_dim"], m["num_key_value_heads"] * m["head_dim"]
        extra_bytes = extra_flops = 0
        width, vocab = m["hidden_size"], m["vocab_size"]
    cached, new = sum(c for c, _ in requests), T
    return {"bytes": e * (body + head) + e * T * width + 2 * e * layers * kv * (cached + new) + 4 * rows * vocab + extra_bytes,
            "flops": 2 * T * body + 2 * rows * head + 4 * layers * heads * d * pairs + extra_flops}


def work(case):
    requests = _requests(case)
    w = _step_work(case, requests)
    for k in range(case.get("new_tokens", 0)):
        s = _step_work(case, [(n + k, 1) for _, n in requests])
        w = {"bytes": w["bytes"] + s["bytes"], "flops": w["flops"] + s["flops"]}
    return w


# ------------------------------------------------------------------------------------------------ inputs

def _gen(seed, name):
    h = hashlib.sha256(f"{seed}:{name}".encode()).digest()
    return torch.Generator(device="cuda").manual_seed(int.from_bytes(h[:8], "little") & 0x7FFFFFFFFFFFFFFF)


def _fill(t, seed, name):
    """The values of the stored tensor `name`.  Llama: matrices as models are initialised, those that add to the residual
    stream scaled down with the depth, and an embedding of the stream's size, so that a layer changes the stream by a part of
    it, as it does in a trained model.  Dizepel: matrices of about unit gain, filters, biases and decays of the size of what
    they join.  Norm weights around one."""
    g, last = _gen(seed, name), name.split(".")[-1]
    if name.startswith("model.") or name.startswith("lm_head"):
        if "norm" in name:
            return t.uniform_(0.8, 1.2, generator=g)
        if "embed" in name:
            return t.normal_(0.0, 1.0, generator=g)
        return t.normal_(0.0, 0.0025 if "o_proj" in name or "down_proj" in name else 0.02, generator=g)
    if last in ("norm", "norm1", "norm2", "norm1b", "norm2b", "out"):
        return t.uniform_(0.7, 1.3, generator=g)
    if last == "A_log":
        return t.uniform_(0.05, 2.05, generator=g).log_()
    if last == "dt_bias":
        return t.normal_(-1.0, 1.0, generator=g)
    if last in ("canon1", "canon2", "conv"):
        return t.normal_(0.0, 0.5, generator=g)
    if last in ("D", "sink", "act", "step", "embed"):
        return t.normal_(0.0, 1.0, generator=g)
    return t.normal_(0.0, 0.5 if t.dim() == 1 else t.shape[1] ** -0.5, generator=g)


def _weight(case, seed, name, *shape):
    """Tensor `name` as the loader would store it, in 64 bits."""
    t = torch.empty(shape, dtype=torch.float32 if _is_kept(name) else DTYPES[case["dtype"]], device="cuda")
    return _fill(t, seed, name).double()


def _is_kept(name):
    """Vectors and short filters that a checkpoint stores, and the engine keeps, in 32 bits (Llama checkpoints have all in 16)."""
    return not name.startswith("model.") and name.split(".")[-1] in (
        "norm", "norm1", "norm2", "norm1b", "norm2b", "out", "canon1", "canon2", "conv", "b", "dt_bias", "A_log", "D", "sink", "act")


def _cached(case, seed, layer, requests):
    """Keys and values of the layer's cached tokens, request after request in whole pages: [pages, 2, kv heads, page, head size]."""
    m = MODELS[case["model"]]
    pages = sum(-(-c // BLOCK) for c, _ in requests)
    t = torch.empty((pages, 2, m["num_key_value_heads"], BLOCK, m["head_dim"]), dtype=DTYPES[case["dtype"]], device="cuda")
    return t.normal_(0.0, 1.0, generator=_gen(seed, f"cache {layer}"))


def _tokens(case, seed, requests):
    """Per request its new tokens of the first step, and of each of the steps after it."""
    m = MODELS[case["model"]]
    g = torch.Generator().manual_seed(seed)
    vocab, more = m.get("vocab_size") or m["vocab"], case.get("new_tokens", CYCLE)
    first = [torch.randint(0, vocab, (n,), generator=g).tolist() for _, n in requests]
    return first, torch.randint(0, vocab, (more, len(requests)), generator=g).tolist()


class _State:
    pass


def _build_model(case, seed):
    """The model on the device, its weights handed to its parts as the loader does."""
    from lmsf_b200 import models  # noqa: F401  (registers the architectures)
    from lmsf_b200.config.registry import resolve_architecture
    from lmsf_b200.parts.decoder import DecoderModel
    from lmsf_b200.weights.loader import collect_requirements
    cfg = dict(MODELS[case["model"]])
    arch, dtype, dev = resolve_architecture(cfg), DTYPES[case["dtype"]], torch.device("cuda:0")
    model = DecoderModel(arch.build_spec(arch.parse_config(cfg)))
    done, per_part, parts = {}, {}, {}
    for part, logical, wspec, names in collect_requirements(model):
        t = done.get(tuple(names))
        if t is None:
            sizes = [wspec.concrete(i) for i in range(len(wspec.shapes))]
            t = torch.empty((sum(s[0] for s in sizes), *sizes[0][1:]), dtype=torch.float32 if _is_kept(names[0]) else dtype, device=dev)
            at = 0
            for name, s in zip(names, sizes):
                _fill(t[at:at + s[0]], seed, name)
                at += s[0]
            done[tuple(names)] = t
        per_part.setdefault(id(part), {})[logical] = t
        parts[id(part)] = part
    for pid, tensors in per_part.items():
        parts[pid].set_weights(tensors)
    model.prepare(dtype, dev)
    return model, dtype, dev


def _seat(s):
    """A cache manager in which the requests hold their cached tokens (the same pages every time)."""
    s.mgr = s.runner.make_cache_manager()
    for i, (cached, _) in enumerate(s.requests):
        s.mgr.add(i)
        if cached:
            s.mgr.reserve(i, cached)
            s.mgr.commit(i, cached)
    s.k = 0


def prepare(case, seed):
    s = _State()
    s.case = case
    from lmsf_b200.engine.model_runner import ModelRunner, StepEntry
    s.Entry, s.requests = StepEntry, _requests(case)
    s.first, s.later = _tokens(case, seed, s.requests)
    model, dtype, dev = _build_model(case, seed)
    grow = case.get("new_tokens", CYCLE)
    pages = sum(-(-(c + n + grow) // BLOCK) for c, n in s.requests) + 8
    s.runner = ModelRunner(model, dtype, dev, BLOCK, num_blocks=pages, max_num_seqs=max(64, len(s.requests)), max_model_len=MAX_LEN[case["model"]])
    if case["kind"] == "step":
        _seat(s)
        if any(c for c, _ in s.requests):
            table = torch.tensor([p for i, (c, _) in enumerate(s.requests) for p in s.mgr.block_table(i, 0)[:-(-c // BLOCK)]], device=dev)
            for layer, cache in enumerate(s.runner.storage.layer_caches):
                cache.kv[table] = _cached(case, seed, layer, s.requests)
    return s


# ------------------------------------------------------------------------------------------------ a pass

def run(s):
    case = s.case
    n = len(s.requests)
    if case["kind"] == "life":
        mgr = s.runner.make_cache_manager()
        for i in range(n):
            mgr.add(i)
        out = [s.runner.step([s.Entry(i, t, [len(t) - 1]) for i, t in enumerate(s.first)], mgr, check=False).clone()]
        for toks in s.later:
            out.append(s.runner.step([s.Entry(i, [t], [0]) for i, t in enumerate(toks)], mgr, check=False).clone())
        for i in range(n):
            mgr.free(i)
        return out
    if case["prompts"]:
        # a prompt runs once: the requests start again from their cached tokens at every pass
        _seat(s)
        return s.runner.step([s.Entry(i, t, [len(t) - 1]) for i, t in enumerate(s.first)], s.mgr, check=False)
    if s.k == CYCLE:
        _seat(s)
    toks = s.later[s.k]
    s.k += 1
    return s.runner.step([s.Entry(i, [t], [0]) for i, t in enumerate(toks)], s.mgr, check=False)


# ------------------------------------------------------------------------------------------------ the same in 64 bits

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _llama_frequencies(m):
    d = m["head_dim"]
    f = m["rope_theta"] ** (-torch.arange(0, d, 2, dtype=torch.float64, device="cuda") / d)
    sc = m.get("rope_scaling")
    if sc:
        turns = sc["original_max_position_embeddings"] * f / (2 * math.pi)
        keep = ((turns - sc["low_freq_factor"]) / (sc["high_freq_factor"] - sc["low_freq_factor"])).clamp(0, 1)
        f = keep * f + (1 - keep) * f / sc["factor"]
    return f


def _turn(x, pos, f, mult=1.0):
    """x [T, heads, d]: value i of the first 2 len(f) turns with value i + len(f) by position * f[i]."""
    n = f.numel()
    ang = pos.double()[:, None, None] * f
    c, s = torch.cos(ang) * mult, torch.sin(ang) * mult
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], -1)


def _attend(q, k, v, first, scale, cap=None, sink=None):
    """q [n, H, d] at positions first.., k and v [keys, G, d] from position 0 -> [n, H, d]; every query sees the keys up to its own."""
    n, H, d = q.shape
    out = torch.empty_like(q)
    group = H // k.shape[1]
    if n == 1 and sink is None:
        s = torch.einsum("ghd,kgd->ghk", q[0].reshape(-1, group, d), k) * scale
        return torch.einsum("ghk,kgd->ghd", torch.softmax(s, -1), v).reshape(1, H, d)
    seen = torch.arange(k.shape[0], device="cuda")[None, :] <= (first + torch.arange(n, device="cuda"))[:, None]
    for h in range(H):
        s = (q[:, h] @ k[:, h // group].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        p = torch.softmax(s, -1)
        out[:, h] = p[:, :k.shape[0]] @ v[:, h // group]
    return out


def _llama_run(case, seed, requests, tokens):
    """Logits of every request's tokens that `want` keeps: the whole new part of each request in one go.  tokens: per request its
    new ids.  Returns per request float64 [new, hidden] before the head, normed."""
    m = MODELS[case["model"]]
    D, d, eps = m["hidden_size"], m["head_dim"], m["rms_norm_eps"]
    H, G, I = m["num_attention_heads"], m["num_key_value_heads"], m["intermediate_size"]
    W = lambda name, *shape: _weight(case, seed, name, *shape)
    f = _llama_frequencies(m)
    lens = [len(t) for t in tokens]
    E = torch.empty((m["vocab_size"], D), dtype=DTYPES[case["dtype"]], device="cuda")
    _fill(E, seed, "model.embed_tokens.weight")
    x = E[torch.tensor([t for ts in tokens for t in ts], device="cuda")].double()
    pos = torch.cat([torch.arange(c, c + n, device="cuda") for (c, _), n in zip(requests, lens)])
    for layer in range(m["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        h = _rms(x, eps) * W(p + "input_layernorm.weight", D)
        q = _turn((h @ W(p + "self_attn.q_proj.weight", H * d, D).T).reshape(-1, H, d), pos, f)
        k = _turn((h @ W(p + "self_attn.k_proj.weight", G * d, D).T).reshape(-1, G, d), pos, f)
        v = (h @ W(p + "self_attn.v_proj.weight", G * d, D).T).reshape(-1, G, d)
        old = _cached(case, seed, layer, requests) if any(c for c, _ in requests) else None
        o, at, page = torch.empty_like(q), 0, 0
        for (c, _), n in zip(requests, lens):
            ks, vs = k[at:at + n], v[at:at + n]
            if c:
                np_ = -(-c // BLOCK)
                kv = old[page:page + np_].permute(1, 0, 3, 2, 4).reshape(2, -1, G, d)[:, :c].double()
                ks, vs = torch.cat([kv[0], ks]), torch.cat([kv[1], vs])
                page += np_
            o[at:at + n] = _attend(q[at:at + n], ks, vs, c, d ** -0.5)
            at += n
        x = x + o.reshape(-1, H * d) @ W(p + "self_attn.o_proj.weight", D, H * d).T
        h = _rms(x, eps) * W(p + "post_attention_layernorm.weight", D)
        g = h @ W(p + "mlp.gate_proj.weight", I, D).T
        g = g * torch.sigmoid(g) * (h @ W(p + "mlp.up_proj.weight", I, D).T)
        x = x + g @ W(p + "mlp.down_proj.weight", D, I).T
    x = _rms(x, eps) * W("model.norm.weight", D)
    head = E.double() if m["tie_word_embeddings"] else W("lm_head.weight", m["vocab_size"], D)
    return list(x.split(lens)), head


def _filter(u, w):
    """u [T, C], w [C, taps]: the sum of w[:, j] * u at (t - taps + 1 + j), nothing before the first token."""
    T, taps = u.shape[0], w.shape[1]
    y = torch.zeros_like(u)
    for j in range(taps):
        back = taps - 1 - j
        if back < T:
            y[back:] += w[:, j] * u[:T - back]
    return y


def _yarn(rot):
    n, base, sc = rot["dims"], rot["base"], rot["scaling"]
    at = lambda turns: n * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), n - 1)
    f = []
    for i in range(n // 2):
        r = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        f.append(base ** (-2.0 * i / n) * (r / sc["factor"] + 1 - r))
    return torch.tensor(f, dtype=torch.float64, device="cuda"), 0.1 * math.log(sc["factor"]) + 1


def _dizepel_run(case, seed, requests, tokens):
    cfg = MODELS["dizepel"]
    D, eps, taps = cfg["width"], cfg["norm"]["eps"], cfg["canon"]["taps"]
    W = lambda name, *shape: _weight(case, seed, name, *shape)
    norm = lambda z, w: _rms(z - z.mean(-1, keepdim=True), eps) * w
    lens = [len(t) for t in tokens]
    x = W("embed", cfg["vocab"], D)[torch.tensor([t for ts in tokens for t in ts], device="cuda")] * cfg["embedding"]["scale"]
    x = x + W("loop.step", 1, D)[0]
    each = lambda u, w: torch.cat([_filter(s, w) for s in u.split(lens)])
    for i, L in enumerate(cfg["layers"]):
        p, a, b = f"l{i}.", L["mixer"]["left"], L["mixer"]["right"]
        l, r = p + "mix.left.", p + "mix.right."
        h = norm(x, W(p + "norm1", D))
        h = h + each(h, W(p + "canon1", D, taps))
        # attention
        H, G, d = a["heads"], a["kv_heads"], a["dim"]
        q = each(h @ W(l + "q", H * d, D).T + W(l + "q.b", H * d), W(l + "q.conv", H * d, a["conv"])).reshape(-1, H, d)
        k = each(h @ W(l + "k", G * d, D).T + W(l + "k.b", G * d), W(l + "k.conv", G * d, a["conv"])).reshape(-1, G, d)
        f, mult = _yarn(a["rot"])
        pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
        qr, kr, sink = _turn(q, pos, f, mult), _turn(k, pos, f, mult), W(l + "sink", H)
        o = torch.cat([_attend(qs, ks, vs, 0, a["scale"], a["softcap"], sink) for qs, ks, vs in zip(qr.split(lens), kr.split(lens), k.split(lens))])
        left = o.reshape(-1, H * d) @ W(l + "o", D, H * d).T
        # state space
        Hs, dv, N, Gs = b["heads"], b["vdim"], b["state"], b["groups"]
        inner, ch = Hs * dv, Hs * dv + 2 * Gs * N
        z, xbc, dt = (h @ W(r + "in", inner + ch + Hs, D).T).split([inner, ch, Hs], -1)
        xbc = each(xbc, W(r + "conv", ch, b["conv"])) + W(r + "conv.b", ch)
        xs, B, C = (xbc * torch.sigmoid(xbc)).split([inner, Gs * N, Gs * N], -1)
        xs = xs.reshape(-1, Hs, dv)
        B, C = (t.reshape(-1, Gs, N).repeat_interleave(Hs // Gs, 1) for t in (B, C))
        step = torch.nn.functional.softplus(dt + W(r + "dt_bias", Hs), threshold=1e9)
        decay, skip = torch.exp(-torch.exp(W(r + "A_log", Hs)) * step), W(r + "D", Hs)
        # the requests side by side, padded to the longest
        y, at = torch.empty_like(xs), 0
        longest, n = max(lens), len(lens)
        pad = lambda t: torch.nn.utils.rnn.pad_sequence(list(t.split(lens)), batch_first=True)
        bx, cx, dx, xx = pad(B * step[..., None]), pad(C), pad(decay), pad(xs)
        S, ys = torch.zeros((n, Hs, N, dv), dtype=torch.float64, device="cuda"), torch.empty_like(xx)
        for t in range(longest):
            S.mul_(dx[:, t, :, None, None]).addcmul_(bx[:, t, :, :, None], xx[:, t, :, None, :])
            ys[:, t] = torch.matmul(cx[:, t, :, None, :], S)[:, :, 0]
        y = torch.cat([ys[j, :lens[j]] for j in range(n)]) + skip[:, None] * xs
        y = y.reshape(-1, inner) * (z * torch.sigmoid(z))
        parts = b["norm_groups"]
        y = _rms(y.reshape(-1, parts, inner // parts), eps).reshape(-1, inner) * W(r + "norm", inner)
        right = y @ W(r + "o", D, inner).T
        x = x + norm(0.5 * (_rms(left, eps) * W(l + "out", D) + _rms(right, eps) * W(r + "out", D)), W(p + "norm1b", D))
        h = norm(x, W(p + "norm2", D))
        h = h + each(h, W(p + "canon2", D, taps))
        ff = L["mlp"]["ff"]
        z = h @ W(p + "mlp.up", ff, D).T
        c = W(p + "mlp.act", 4)
        x = x + norm((c[0] * _rms(z, eps) + c[1] * _rms(z ** 2, eps) + c[2] * _rms(z ** 3, eps) + c[3]) @ W(p + "mlp.down", D, ff).T,
                     W(p + "norm2b", D))
    return list(norm(x, W("final.norm", D)).split(lens)), W("head", cfg["vocab"], D)


def exact(case, seed):
    with torch.no_grad():
        requests = _requests(case)
        first, later = _tokens(case, seed, requests)
        model = _dizepel_run if case["model"] == "dizepel" else _llama_run
        if case["kind"] == "life":
            # the whole of every request at once: each token sees what came before it, as it does step by step
            whole = [t + [row[i] for row in later] for i, t in enumerate(first)]
            hidden, head = model(case, seed, requests, whole)
            at = lambda k: torch.stack([h[len(t) - 1 + k] for h, t in zip(hidden, first)])
            return [at(k) @ head.T for k in range(len(later) + 1)]
        new = first if case["prompts"] else [[t] for t in later[0]]
        hidden, head = model(case, seed, requests, new)
        return torch.stack([h[-1] for h in hidden]) @ head.T


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 1e-4}           # against 64 bits: 1.2e-6
    return {"rel": 0.02, "max": 0.15}               # against 64 bits: 0.002 to 0.008; two implementations: 1.4 times that
