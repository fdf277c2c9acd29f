"""What a user of this engine has it do, as cases to time and to compare.

Every case is one step of ``ModelRunner``, the step function that ``LLMEngine`` and ``bin/trace_run`` drive: prompts,
portions of long prompts, single tokens behind a context, and mixtures of them, through one or more layers of a named
design.  Two cases are whole Qwen2.5-1.5B models (the benchmark's headline shape); the others are single layers of the
designs at the named shapes' sizes, between an embedding and a head, so that each kind of mixer and feed-forward is seen by
itself.  Where the step returns logits at every place (as a trace replay asks for) the vocabulary is cut to 1,024 entries:
the layer is what is looked at, not the head.

A case: ``model`` (a named shape), ``layer`` ("" for the shape's own layers, else "<mixer type>+<feed-forward kind>": a
model of such layers alone), ``layers`` (how many), ``vocab`` (0: the shape's), ``dtype``, ``new`` (the tokens that each
request brings, "2048" or "391,130,1"), ``behind`` (the tokens of each that the cache already holds), ``want`` ("last" or
"all": the places whose logits come back), ``sampled`` (single-token steps: temperature, top-k and top-p instead of
the largest logit).
"""

import math
import zlib

import torch
import torch.nn.functional as F

DEV = "cuda:0"
PAGE = 16          # tokens a page (the engine's default)
PORTION = 2048     # how long prompts are brought in
CUT_VOCAB = 1024


def _case(name, model, layer, layers, vocab, new, behind, want, dtype="bfloat16", sampled=False):
    return dict(name=name, model=model, layer=layer, layers=layers, vocab=vocab, dtype=dtype, new=new, behind=behind, want=want,
                sampled=sampled)


def listed():
    ragged = [1024 + (37 * i * i + 211 * i) % 1024 for i in range(64)]
    return [
        # the headline: a chat server's steady state at a small batch, the whole model, greedy
        _case("decode_8", "qwen2.5-1.5b", "", 28, 0, _list([1] * 8), _list([1024] * 8), "last"),
        # a busy server with the sampler on: 64 requests of different lengths, a wide layer, the full vocabulary
        _case("decode_64_sampled", "qwen2.5-7b", "", 1, 0, _list([1] * 64), _list(ragged), "last", sampled=True),
        # a prompt of ordinary length through the whole model: the time to the first token
        _case("prompt_2048", "qwen2.5-1.5b", "", 28, 0, "2048", "0", "last"),
        # a late portion of a long document, not a multiple of anything: attention over a long cache
        _case("long_prompt_portion", "qwen2.5-1.5b", "", 1, CUT_VOCAB, "2003", "13001", "all"),
        # continuous batching: two new prompts' portions ride with 24 requests that decode, a wide layer
        _case("mixed_step", "qwen2.5-7b", "", 1, CUT_VOCAB, _list([391, 130] + [1] * 24), _list([0, 517] + ragged[:24]), "all"),
        # the float32 path, which results are checked against: a short prompt behind a short context
        _case("float32_prompt", "qwen2.5-1.5b", "", 1, CUT_VOCAB, "200", "120", "all", dtype="float32"),
        # routed experts beside latent attention: a prompt
        _case("experts_prompt", "rapitar-2k", "latent_attention+moe", 1, CUT_VOCAB, "2048", "0", "all"),
        # the same layer while it decodes for a few requests
        _case("experts_decode", "rapitar-2k", "latent_attention+moe", 1, CUT_VOCAB, _list([1] * 8), _list([1024] * 8), "all"),
        # attention over a sliding window that keeps the first positions: prompts of three requests, ragged
        _case("window_prompts", "dezolorn-2k", "attention+dense", 1, CUT_VOCAB, "1500,421,127", "0,0,0", "all"),
        # the delta rule over a prompt
        _case("delta_prompt", "dezolorn-2k", "delta+dense", 1, CUT_VOCAB, "1024", "0", "all"),
        # a state-space layer over ragged prompts
        _case("state_space_prompts", "rapitar-2k", "mamba2+dense", 1, CUT_VOCAB, "900,333,65", "0,0,0", "all"),
        # the smallest call: a recurrent layer while it decodes for two requests, where launches are what counts
        _case("retention_decode", "dezolorn-2k", "retention+dense", 1, CUT_VOCAB, "1,1", "96,41", "all"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def split(total, parts):
        cuts = sorted(rng.sample(range(1, total), parts - 1)) if parts > 1 else []
        return [b - a for a, b in zip([0] + cuts, cuts + [total])]

    kind = rng.choice(("decode", "prompt", "portion", "mixed", "float32", "listed_prompt", "listed_prompt", "listed_decode"))
    qwen = rng.choice(("qwen2.5-1.5b", "qwen2.5-7b"))
    if kind == "decode":
        n = log(1, 64)
        return _drawn(qwen, "", rng.choice((1, 2)), 0, [1] * n, [log(64, 3000) for _ in range(n)], "last", sampled=rng.random() < 0.4)
    if kind == "prompt":
        total = log(24, 3000)
        new = split(total, min(rng.randint(1, 5), total))
        return _drawn(qwen, "", rng.choice((1, 2)), CUT_VOCAB, new, [0] * len(new), "all")
    if kind == "portion":
        return _drawn("qwen2.5-1.5b", "", 1, CUT_VOCAB, [log(128, 2048)], [log(1024, 12000)], "all")
    if kind == "mixed":
        n, portions = log(2, 48), rng.randint(1, 3)
        new = [log(16, 500) for _ in range(portions)] + [1] * n
        return _drawn(qwen, "", 1, CUT_VOCAB, new, [log(1, 1000) for _ in range(portions)] + [log(64, 2500) for _ in range(n)], "all")
    if kind == "float32":
        return _drawn("qwen2.5-1.5b", "", 1, CUT_VOCAB, [log(1, 300)], [log(16, 600)], "all", dtype="float32")
    model, layer = rng.choice((("rapitar-2k", "latent_attention+moe"), ("rapitar-2k", "mamba2+dense"), ("rapitar-2k", "mamba2+moe"),
                               ("dezolorn-2k", "attention+dense"), ("dezolorn-2k", "delta+dense"), ("dezolorn-2k", "retention+dense")))
    if kind == "listed_prompt":
        total = log(48, 2048)
        new = split(total, min(rng.randint(1, 4), total))
        return _drawn(model, layer, 1, CUT_VOCAB, new, [0] * len(new), "all")
    n = log(1, 32)
    return _drawn(model, layer, 1, CUT_VOCAB, [1] * n, [log(16, 1000) for _ in range(n)], "all")


def _drawn(*args, **kwargs):
    model, layer, layers, vocab, new, behind, want = args
    case = _case("", model, layer, layers, vocab, _list(new), _list(behind), want, **kwargs)
    del case["name"]
    return case


def _list(numbers):
    return ",".join(str(n) for n in numbers)


def _numbers(text):
    return [int(n) for n in text.split(",")]


# ---- the model, its weights and its tokens --------------------------------------------------------------------------
def _config(case):
    from clockwork_b200 import models  # noqa: F401  (registers the designs and their named shapes)
    from clockwork_b200.config.registry import shape_config

    if case["layer"]:
        raw = shape_config(case["model"])
        mixer, ffn = case["layer"].split("+")
        layer = next(x for x in raw["layers"] if x["type"] == mixer and (x["mlp"] or {}).get("kind") == ffn)
        raw["layers"] = [layer] * case["layers"]
        raw["vocab"] = case["vocab"] or raw["vocab"]
    else:
        raw = shape_config(case["model"], case["layers"])
        raw["vocab_size"] = case["vocab"] or raw["vocab_size"]
    return raw


def _vocab(raw):
    return raw.get("vocab_size") or raw["vocab"]


def _draw_tensor(name, shape, role, init, dtype, seed):
    """Weights as a model of the design starts out: products that keep the scale of what they are given, decays and step
    sizes spread as in published state-space models."""
    gen = torch.Generator(device=DEV).manual_seed((seed << 32) ^ zlib.crc32(name.encode()))
    t = torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0.0, 1.0, generator=gen)
    last = name.rsplit(".", 1)[-1]
    if last == "A_log":
        t = torch.special.ndtr(t).mul_(15.0).add_(1.0).log_()                      # decay rates from 1 to 16
    elif last == "dt_bias":
        dt = torch.exp(torch.special.ndtr(t) * math.log(100.0) + math.log(1e-3))   # step sizes from 0.001 to 0.1
        t = dt + torch.log(-torch.expm1(-dt))                                      # what softplus maps to them
    elif last == "conv":
        t.mul_(shape[-1] ** -0.5)
    elif init == "norm":
        t.mul_(0.1).add_(1.0)
    elif init == "zeros":
        t.mul_(0.1)                                                                # (norms stored as the distance from one)
    elif init in ("bias", "embedding"):
        t.mul_(0.02)
    else:
        t.mul_(shape[-1] ** -0.5)
    return t.to(dtype if role in ("matrix", "table") else torch.float32)


def _weights(case, raw, seed, decls):
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    by_name = {d.name: d for d in decls}

    def fetch(name):
        d = by_name[name]
        return _draw_tensor(name, d.shape, d.role, d.init, dtype, seed)

    return fetch


def _tokens(case, vocab, seed):
    """Per request: (the tokens that its cache holds, the tokens that it brings)."""
    out = []
    for i, (new, behind) in enumerate(zip(_numbers(case["new"]), _numbers(case["behind"]))):
        gen = torch.Generator().manual_seed(seed * 1000 + i)
        ids = torch.randint(0, vocab, (behind + new,), generator=gen).tolist()
        out.append((ids[:behind], ids[behind:]))
    return out


def _wanted(case, new):
    return list(range(new)) if case["want"] == "all" else [new - 1]


# ---- one step --------------------------------------------------------------------------------------------------------
class _Step:
    pass


def prepare(case, seed):
    """A loaded model, its cache with the requests' contexts in it, and the step's tokens."""
    from clockwork_b200.cache import CacheManager
    from clockwork_b200.config.registry import spec_from_raw
    from clockwork_b200.engine import ModelRunner, StepEntry
    from clockwork_b200.parts.model import build_model

    raw = _config(case)
    model = build_model(spec_from_raw(raw), torch.float32 if case["dtype"] == "float32" else torch.bfloat16, DEV)
    model.load_weights(_weights(case, raw, seed, model.tensor_decls()))
    tokens = _tokens(case, _vocab(raw), seed)
    pages = sum((len(b) + len(n)) // PAGE + 2 for b, n in tokens)
    s = _Step()
    s.cache = CacheManager(model.cache_needs(), num_pages=pages + pages // 50 + 16, page_size=PAGE, dtype=model.dtype, device=DEV,
                           num_state_slots=len(tokens) + 1)
    s.runner = ModelRunner(model, s.cache)
    s.runner.enable_graphs(max_ctx=max(4096, max(len(b) + len(n) for b, n in tokens) + 1), max_batch=max(8, len(tokens)))
    s.entries, s.positions = [], {}
    for i, (behind, new) in enumerate(tokens):
        rid = f"r{i}"
        if behind:
            s.cache.open(rid)
            for at in range(0, len(behind), PORTION):
                s.runner.step([StepEntry(rid, behind[at : at + PORTION], [])])
            s.positions[rid] = len(behind)
        s.entries.append(StepEntry(rid, new, _wanted(case, len(new))))
    s.fresh = [e.request_id for e in s.entries if e.request_id not in s.positions]
    s.single = bool(s.positions) and not s.fresh and all(len(e.tokens) == 1 for e in s.entries)
    s.sampling = [(0.8, 50, 0.9, seed + i, 7) for i in range(len(tokens))] if case["sampled"] else None
    return s


def run(s):
    """The step.  Requests without a context are opened for it and closed behind it; the others stand where their context
    ends again afterwards (a recurrent layer's state goes on)."""
    for rid in s.fresh:
        s.cache.open(rid)
    if s.single:
        tokens = s.runner.decode_with_graph(s.entries, s.sampling)
        out = {"logits": s.runner.last_graph.logits[: len(s.entries)], "tokens": tokens}
    else:
        out = {"logits": s.runner.step(s.entries)}
    for rid in s.fresh:
        s.cache.close(rid)
    for rid, position in s.positions.items():
        s.cache.get(rid).num_computed = position
    return out


# ---- what a step cannot do without -----------------------------------------------------------------------------------
def _mixer_shape(raw, mixer):
    """(kind, numbers cached per token, multiply-adds per (token, key), window or None, numbers of state, multiply-adds of a
    state's update and read-out per token)."""
    if mixer is None:
        heads, kv = raw["num_attention_heads"], raw["num_key_value_heads"]
        dim = raw.get("head_dim") or raw["hidden_size"] // heads
        return 2 * kv * dim, 2 * heads * dim, None, 0, 0
    kind, m = mixer
    if kind == "latent_attention":  # (with keys and values made per head: the fewest operations for a prompt)
        return m["kv_rank"] + m["rot_dim"], m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), None, 0, 0
    if kind == "attention":
        return (m["dim"] + m["vdim"]) * m["kv_heads"], m["heads"] * (m["dim"] + m["vdim"]), m["mask"]["size"] + m["mask"]["keep_first"], 0, 0
    if kind == "mamba2":
        s = m["heads"] * m["state"] * m["vdim"]
        return 0, 0, None, s, 2 * s
    s = m["heads"] * m["dim"] * m["vdim"]
    return 0, 0, None, s, (3 if kind == "delta" else 2) * s


def work(case):
    from clockwork_b200.config.registry import spec_from_raw
    from clockwork_b200.parts.model import tensor_decls_for_spec

    raw = _config(case)
    new, behind = _numbers(case["new"]), _numbers(case["behind"])
    tokens, size = sum(new), 4 if case["dtype"] == "float32" else 2
    rows = tokens if case["want"] == "all" else len(new)
    vocab = _vocab(raw)
    width = raw.get("hidden_size") or raw["width"]
    bytes_, flops = vocab * width * size + tokens * width * size, 2 * rows * vocab * width
    bytes_ += rows * vocab * 4
    for d in tensor_decls_for_spec(spec_from_raw(raw)):
        if d.role not in ("matrix", "table") or d.name in ("embed", "head", "model.embed_tokens.weight", "lm_head.weight"):
            continue
        share, used = 1.0, 1.0
        if ".mlp.e" in d.name:  # one expert of many: the share of tokens that go there, and the chance that any does
            router = raw["layers"][0]["mlp"]["router"]
            share = router["top"] / router["experts"]
            used = 1.0 - (1.0 - share) ** tokens
        numbers = math.prod(d.shape)
        bytes_ += numbers * size * used
        if not d.name.endswith(".conv"):
            flops += 2 * numbers * tokens * share
    for layer in raw["layers"] if case["layer"] else [None] * case["layers"]:
        row, per_key, window, state, update = _mixer_shape(raw, None if layer is None else (layer["type"], layer["mixer"]))
        for n, b in zip(new, behind):
            keys = sum(min(b + i + 1, window or b + n) for i in range(n))
            flops += 2 * per_key * keys + 2 * update * n
            bytes_ += row * size * ((min(b, window or b) if row else 0) + n) + 4 * state * (2 if b else 1)
    return {"bytes": float(bytes_), "flops": float(flops)}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}  # (2e-6 to 4e-6 from the result in 64 bits)
    # 16-bit activations between the kernels of a layer: their rounding is what two correct implementations differ by (one
    # layer is 0.0025 to 0.0075 from the result in 64 bits, 28 layers 0.009)
    layers = case["layers"]
    t = {"rel": 1.5e-2 if layers <= 2 else 3e-2, "max": 0.15 if layers <= 2 else 0.3}
    if _numbers(case["new"]) == [1] * len(_numbers(case["new"])) and min(_numbers(case["behind"])) > 0:
        t["differ"] = 0.6  # tokens: the largest of many close logits, and draws between close sums
    return t


# ---- the same in 64 bits, from the equations -------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, eps):
    x = x - x.mean(-1, keepdim=True)
    return _rms(x, eps) * w


def _frequencies(dims, base, scaling):
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEV)
    f = base ** (-2.0 * i / dims)
    if scaling is None:
        return f, 1.0
    at = lambda turns: dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f * (ramp / scaling["factor"] + 1 - ramp), 1 + 0.1 * math.log(scaling["factor"])


def _rotate(x, base, dims, scaling=None, interleaved=False):
    """x [T, heads, d], row t at position t: the first ``dims`` entries of every head."""
    f, amplitude = _frequencies(dims, base, scaling)
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=DEV)[:, None] * f
    cos, sin = (angle.cos() * amplitude)[:, None], (angle.sin() * amplitude)[:, None]
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if interleaved else (x[..., : dims // 2], x[..., dims // 2 : dims])
    turned = (a * cos - b * sin, b * cos + a * sin)
    turned = torch.stack(turned, -1).flatten(-2) if interleaved else torch.cat(turned, -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _attend(q, k, v, scale, start, visible=None, sink=None):
    """q [T, H, dk], k [T, G, dk], v [T, G, dv] of one request -> [T - start, H, dv], rows from ``start`` on."""
    t, heads, _ = q.shape
    per = heads // k.shape[1]
    out = []
    for a in range(start, t, 256):
        b = min(a + 256, t)
        i, j = torch.arange(a, b, device=DEV)[:, None], torch.arange(b, device=DEV)[None, :]
        seen = (j <= i) if visible is None else (j <= i) & visible(i, j)
        rows = []
        for h in range(heads):
            s = (q[a:b, h] @ k[:b, h // per].T * scale).masked_fill(~seen, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[h].expand(b - a, 1)], 1)
            rows.append(torch.softmax(s, -1)[:, :b] @ v[:b, h // per])
        out.append(torch.stack(rows, 1))
    return torch.cat(out)


def _conv(x, w, b=None):
    t, taps = x.shape[0], w.shape[1]
    padded = F.pad(x, (0, 0, taps - 1, 0))
    y = sum(padded[j : j + t] * w[:, j] for j in range(taps))
    return F.silu(y if b is None else y + b)


def _scan(q, k, v, decay, beta=None):
    """q, k [T, H, dk], v [T, H, dv], decay [T, H]; with ``beta`` [T, H] the delta rule."""
    state = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=torch.float64, device=DEV)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        state = state * decay[t][:, None, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", state, k[t]))
        state = state + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", state, q[t])
    return out


def _mix(raw, layer, h, w, p, start):
    """The mixer of one request's rows (a whole sequence), rows from ``start`` on (recurrent ones: all rows)."""
    t = h.shape[0]
    if layer is None:
        heads, kv = raw["num_attention_heads"], raw["num_key_value_heads"]
        dim = raw.get("head_dim") or raw["hidden_size"] // heads
        q, k, v = ((h @ w(f"{p}.self_attn.{n}_proj.weight").T + w(f"{p}.self_attn.{n}_proj.bias")).view(t, -1, dim) for n in "qkv")
        q, k = (_rotate(x, raw["rope_theta"], dim) for x in (q, k))
        return _attend(q, k, v, dim ** -0.5, start).flatten(1) @ w(f"{p}.self_attn.o_proj.weight").T
    kind, m, eps, p = layer["type"], layer["mixer"], raw["norm"]["eps"], f"{p}.mix"
    if kind == "latent_attention":
        heads, dim, rot, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        q = ((_rms(h @ w(f"{p}.dq").T, eps) * w(f"{p}.dq.norm")) @ w(f"{p}.uq").T).view(t, heads, dim + rot)
        q = torch.cat([q[..., :dim], _rotate(q[..., dim:], m["rot"]["base"], rot)], -1)
        down = h @ w(f"{p}.dkv").T
        c = _rms(down[:, :rank], eps) * w(f"{p}.dkv.norm")
        shared = _rotate(down[:, None, rank:], m["rot"]["base"], rot).expand(t, heads, rot)
        k = torch.cat([(c @ w(f"{p}.uk").T).view(t, heads, dim), shared], -1)
        v = (c @ w(f"{p}.uv").T).view(t, heads, m["vdim"])
        o = _attend(q, k, v, m["scale"], start, sink=w(f"{p}.sink")).flatten(1)
        return (o * torch.sigmoid(h[start:] @ w(f"{p}.g").T)) @ w(f"{p}.o").T
    if kind == "attention":
        q, k = ((_rms(h @ w(f"{p}.{n}").T, eps) * w(f"{p}.{n}.norm")).view(t, -1, m["dim"]) for n in "qk")
        v = (h @ w(f"{p}.v").T).view(t, -1, m["vdim"])
        q, k = (_rotate(x, m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"], True) for x in (q, k))
        seen = lambda i, j: (i - j < m["mask"]["size"]) | (j < m["mask"]["keep_first"])  # noqa: E731
        return _attend(q, k, v, m["scale"], start, seen).flatten(1) @ w(f"{p}.o").T
    if kind == "mamba2":
        heads, vdim, n, groups = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = heads * vdim
        z, xbc, dt = (h @ w(f"{p}.in").T).split([inner, inner + 2 * groups * n, heads], 1)
        x, b, c = _conv(xbc, w(f"{p}.conv"), w(f"{p}.conv.b")).split([inner, groups * n, groups * n], 1)
        x = x.view(t, heads, vdim)
        b, c = (y.view(t, groups, n).repeat_interleave(heads // groups, 1) for y in (b, c))
        dt = F.softplus(dt + w(f"{p}.dt_bias"), threshold=1e9)
        y = _scan(c, b, x * dt[..., None], torch.exp(-torch.exp(w(f"{p}.A_log")) * dt)) + w(f"{p}.D")[:, None] * x
        y = (y.reshape(t, inner) * F.silu(z)).view(t, m["norm_groups"], -1)
        return (_rms(y, eps).reshape(t, inner) * w(f"{p}.norm")) @ w(f"{p}.o").T
    heads, dim, vdim = m["heads"], m["dim"], m["vdim"]
    if kind == "retention":
        q, k, v = ((h @ w(f"{p}.{n}").T).view(t, heads, -1) for n in "qkv")
        q, k = (_rotate(x, m["rot"]["base"], m["rot"]["dims"]) for x in (q, k))
        decay = torch.tensor(m["decay"], dtype=torch.float32, device=DEV).double().expand(t, heads)
        o = _rms(_scan(q, k * dim ** -0.5, v, decay), eps).reshape(t, -1)
        return (o * F.silu(h @ w(f"{p}.g").T)) @ w(f"{p}.o").T
    q, k, v = (_conv(h @ w(f"{p}.{n}").T, w(f"{p}.{n}.conv")).view(t, -1, d) for n, d in (("q", dim), ("k", dim), ("v", vdim)))
    q, k = ((x / torch.sqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(heads // m["kv_heads"], 1) for x in (q, k))
    decay = torch.exp(-torch.exp(w(f"{p}.A_log")) * F.softplus(h @ w(f"{p}.a").T + w(f"{p}.dt_bias"), threshold=1e9))
    o = _scan(q * dim ** -0.5, k, v, decay, torch.sigmoid(h @ w(f"{p}.b").T))
    o = _rms(o, eps) * w(f"{p}.norm") * F.silu(h @ w(f"{p}.g").T).view(t, heads, vdim)
    return o.reshape(t, -1) @ w(f"{p}.o").T


def _feed(raw, layer, h, w, p):
    if layer is None or raw.get("architecture") == "Dezolorn":
        names = [f"{p}.mlp.{n}_proj.weight" if layer is None else f"{p}.mlp.{n}" for n in ("gate", "up", "down")]
        gate, up, down = (w(n).T for n in names)
        return (F.silu(h @ gate) * (h @ up)) @ down
    if layer["mlp"]["kind"] == "dense":
        return F.gelu(h @ w(f"{p}.mlp.up").T, approximate="tanh") @ w(f"{p}.mlp.down").T
    router = layer["mlp"]["router"]
    # (the logits are ranked from the rounded rows, as a 16-bit run has them: a choice is not a rounding error)
    values, chosen = torch.topk(h @ w(f"{p}.mlp.router").T + w(f"{p}.mlp.router.b"), router["top"], -1)
    share, out = torch.softmax(values, -1), torch.zeros_like(h)
    for e in range(router["experts"]):
        row, place = (chosen == e).nonzero(as_tuple=True)
        if len(row):
            x = h[row]
            y = (F.silu(x @ w(f"{p}.mlp.e{e}.gate").T) * (x @ w(f"{p}.mlp.e{e}.up").T)) @ w(f"{p}.mlp.e{e}.down").T
            out.index_add_(0, row, y * share[row, place][:, None])
    return out


def exact(case, seed):
    from clockwork_b200.config.registry import spec_from_raw
    from clockwork_b200.parts.model import tensor_decls_for_spec

    raw = _config(case)
    fetch = _weights(case, raw, seed, tensor_decls_for_spec(spec_from_raw(raw)))
    w = lambda name: fetch(name).double()  # noqa: E731
    qwen = not case["layer"]
    requests = _tokens(case, _vocab(raw), seed)
    table = fetch("model.embed_tokens.weight" if qwen else "embed")
    xs = [table[torch.tensor(b + n, device=DEV)].double() for b, n in requests]
    eps = raw["rms_norm_eps"] if qwen else raw["norm"]["eps"]

    def norm(x, name):
        if qwen:
            return _rms(x, eps) * w(f"{name}.weight")
        return _rms(x, eps) * (1 + w(name)) if raw["architecture"] == "Rapitar" else _layer_norm(x, w(name), eps)

    for i in range(case["layers"]):
        layer = None if qwen else raw["layers"][i]
        p = f"model.layers.{i}" if qwen else f"l{i}"
        kept = {}

        def weight(name):  # every tensor drawn once a layer
            if name not in kept:
                kept[name] = w(name)
            return kept[name]

        recurrent = layer is not None and "attention" not in layer["type"]
        first, second = ("input_layernorm", "post_attention_layernorm") if qwen else ("norm1", "norm2")
        last = i == case["layers"] - 1
        # (rows that only feed the others as keys are not carried through the last layer)
        starts = [len(b) if last else 0 for b, _ in requests]
        hs = [norm(x, f"{p}.{first}") for x in xs]
        mixed = [_mix(raw, layer, h, weight, p, 0 if recurrent else a)[a if recurrent else 0 :] for h, a in zip(hs, starts)]
        xs = [x[a:] for x, a in zip(xs, starts)]
        lens = [len(x) for x in xs]
        if not qwen and raw["architecture"] == "Rapitar":  # mixer and feed-forward side by side behind one norm
            h = torch.cat([h[a:] for h, a in zip(hs, starts)])
            if layer["mlp"]["kind"] == "moe" and case["dtype"] == "bfloat16":
                h = h.to(torch.bfloat16).double()
            x = torch.cat(xs) + torch.cat(mixed) + _feed(raw, layer, h, weight, p)
        else:
            x = torch.cat(xs) + torch.cat(mixed)
            x = x + _feed(raw, layer, norm(x, f"{p}.{second}"), weight, p)
        xs = list(x.split(lens))
        del hs, mixed, x
    rows = torch.cat([x[torch.tensor(_wanted(case, len(n)), device=DEV)] for x, (_, n) in zip(xs, requests)])
    if qwen:
        head = w("model.embed_tokens.weight" if raw.get("tie_word_embeddings") else "lm_head.weight")
        logits = norm(rows, "model.norm") @ head.T
    else:
        logits = norm(rows, "final.norm") @ w("head").T
        if raw.get("logit_softcap"):
            cap = raw["logit_softcap"]
            logits = cap * torch.tanh(raw.get("logit_scale", 1.0) * logits / cap)
    out = {"logits": logits}
    if min(_numbers(case["behind"])) > 0 and set(_numbers(case["new"])) == {1}:
        out["tokens"] = None
    return out
