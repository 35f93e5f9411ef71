"""What a program does with this framework, as cases that can be timed and compared: single layers of the engine's
designs through their parts' ``forward``, and a whole prompt through ``Engine.step``.

A case names a kind of layer at the sizes of one of the framework's benchmark configurations and a step: ``requests``
requests that bring ``tokens`` tokens each behind ``cached`` ones (``ragged``: each request brings and holds fewer than the
one before).  Steps of one token per request replay a recording of the layer, as the engine replays its decode steps; other
steps are launched, as the engine launches a prompt's.  ``exact`` states each layer in plain torch in 64 bits.
"""

from __future__ import annotations

import math
import zlib

import torch

from yalis_b200.config.presets import preset
from yalis_b200.config.registry import parse_config
from yalis_b200.engine.context import HostStep, StepContext
from yalis_b200.engine.engine import Engine, StepEntry
from yalis_b200.parts.base import PagedKVCache, ResidualStream, SlotStateCache, build_block, make_part

DEV = "cuda:0"
GROUP = "kv"
# kind -> (configuration, layer, place of the part in the layer, part inside a sum of mixers)
KINDS = {
    "block": ("Llama-3.2-1B", 0, None, None),               # norm, attention, norm, gated feed-forward
    "block_8b": ("Llama-3-8B", 0, None, None),
    "attention_window": ("vepivik-1b", 0, "mixer", None),   # a sliding window, no positions in the scores
    "attention_chunk": ("sazavik-1b", 2, "mixer", None),    # chunks, interleaved rotation, learned sinks, a gate
    "attention_slopes": ("sazavik-1b", 1, "mixer", None),   # a window, biases, a distance bias, a gate
    "latent_window": ("vepivik-1b", 1, "mixer", None),      # 256 + 64 sizes, YaRN, a gate
    "latent_sink": ("pametar-1b", 1, "mixer", None),        # a latent for the queries too, sinks
    "latent_wide": ("vepivik-3b", 1, "mixer", None),        # 24 heads, 384 + 64 sizes
    "delta": ("tirezen-1b", 0, "mixer", None),              # gated delta rule, a decay per head
    "delta_channel": ("tirezen-1b", 1, "mixer", "right"),   # a decay per head and key channel
    "general_delta": ("pametar-1b", 0, "mixer", None),
    "retention": ("tirezen-1b", 2, "mixer", None),
    "lightning": ("lagulorn-1b", 0, "mixer", None),
    "state_space": ("ludelorn-1b", 0, "mixer", "right"),
    "experts": ("vepivik-1b", 0, "feed_forward", None),     # 16 experts, 2 chosen, squared relu, a shared expert
    "experts_gated": ("pametar-1b", 0, "feed_forward", None),
    "whole": ("Llama-3.2-1B", None, None, None),            # a prompt to its last logits, through WHOLE_LAYERS layers
}
WHOLE_LAYERS = 4            # more of them carry bfloat16's roundings past what two correct engines would agree to
RECURRENT = ("delta", "delta_channel", "general_delta", "retention", "lightning", "state_space")
PAGED = ("block", "block_8b", "attention_window", "attention_chunk", "attention_slopes", "latent_window", "latent_sink", "latent_wide")


def _case(kind, requests, tokens, cached, ragged=False, dtype="bfloat16", page=64, name=None):
    c = {"kind": kind, "requests": requests, "tokens": tokens, "cached": cached, "ragged": ragged, "dtype": dtype, "page": page}
    return c if name is None else {**c, "name": name}


def listed():
    return [
        # time to the first token of one request of middling length: the engine's step with its bookkeeping, embedding,
        # layers, output matrix
        _case("whole", 1, 1023, 0, name="whole prompt"),
        # the headline workload's layer: 8 requests decode behind 1,024-token prompts
        _case("block_8b", 8, 1, 1024, page=16, name="block decode"),
        # a layer on the true 32-bit path, as trace replay and validation run it
        _case("block", 1, 250, 0, dtype="float32", name="block float32"),
        # a prompt of the benchmark's length through attention with chunks, sinks and a gate
        _case("attention_chunk", 1, 2048, 0, name="attention prompt"),
        # a busy server's decode step: 64 requests, windowed attention
        _case("attention_window", 64, 1, 1024, True, name="attention decode"),
        # latent attention: a prompt, and a decode step of few requests
        _case("latent_window", 1, 2048, 0, name="latent prompt"),
        _case("latent_sink", 8, 1, 1024, name="latent decode"),
        # the recurrences: one long prompt, unequal prompts side by side, a busy server's decode step
        _case("delta", 1, 2048, 0, name="delta prompt"),
        _case("lightning", 4, 901, 0, True, name="lightning prompts"),
        _case("general_delta", 64, 1, 1024, name="general delta decode"),
        # routed experts: a prompt and the smallest step that is worth batching
        _case("experts", 1, 2048, 0, name="experts prompt"),
        _case("experts_gated", 8, 1, 1024, name="experts decode"),
    ]


def draw(rng):
    kind = rng.choice(["block", "block_8b", "attention_window", "attention_chunk", "attention_slopes", "latent_window", "latent_sink",
                       "latent_wide", "delta", "delta_channel", "general_delta", "retention", "lightning", "state_space", "experts",
                       "experts_gated", "whole"])
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "whole":
        return _case(kind, 1, spread(17, 1000), 0)
    if rng.random() < 0.12:
        return _case(kind, 1, spread(3, 130), rng.choice([0, spread(1, 400)]), dtype="float32", page=rng.choice([16, 64]))
    if rng.random() < 0.5:
        return _case(kind, spread(1, 64), 1, spread(30, 1900), rng.random() < 0.5, page=rng.choice([16, 64]))
    requests = rng.choice([1, 1, 1, 2, 3, 4])
    return _case(kind, requests, spread(17, 4096 // requests if requests > 1 else 2048), rng.choice([0, 0, spread(20, 1000)]),
                 requests > 1 and rng.random() < 0.7, page=rng.choice([16, 64]))


# ---- the step -------------------------------------------------------------------------------------------------------

def _lens(case):
    """(tokens brought, tokens held before) of every request."""
    r, t, c = case["requests"], case["tokens"], case["cached"]
    if not case["ragged"]:
        return [t] * r, [c] * r
    return [max(1, t - i * (t // (2 * r)) - i) if t > 1 else 1 for i in range(r)], [max(0, c - i * (c // (2 * r))) for i in range(r)]


def _decode(case):
    return case["tokens"] == 1 and case["kind"] != "whole"


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _context(case, gen):
    q_lens, before = _lens(case)
    page, n, r = case["page"], sum(q_lens), len(q_lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos, req, starts = [], [], [0]
    for i, (q, b) in enumerate(zip(q_lens, before)):
        pos += range(b, b + q)
        req += [i] * q
        starts.append(starts[-1] + q)
    held = [b + q for q, b in zip(q_lens, before)]
    per = [-(-h // page) for h in held]
    perm = torch.randperm(sum(per) + 2, generator=gen, device=DEV).to(torch.int32)
    table, at = torch.full((r, max(per)), -1, dtype=torch.int32, device=DEV), 0
    for i, p in enumerate(per):
        table[i, :p] = perm[at:at + p]
        at += p
    host = HostStep(slots=list(range(r)), q_start=starts, ctx_before=before, max_q_len=max(q_lens), max_kv_len=max(held))
    return StepContext(n_tokens=n, n_requests=r, token_ids=i32([0] * n), positions=i32(pos), req_of_token=i32(req),
                       q_start=i32(starts), kv_len=i32(held), slots=i32(list(range(r))), logit_rows=i32([]),
                       block_tables={GROUP: table}, host=host, error_flag=torch.zeros(1, dtype=torch.int32, device=DEV),
                       decode_only=max(q_lens) == 1), sum(per) + 2


# ---- weights and inputs, made from the seed ---------------------------------------------------------------------------

def _generator(seed, name):
    gen = torch.Generator(device=DEV)
    gen.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (2 ** 63))
    return gen


def _tensor(name, ps, seed, dtype):
    """A weight as models have it: matrices N(0, 0.02), the recurrences' decays and step sizes spread as they are
    initialised in training (rates of 1 to 16, steps of 0.001 to 0.1), norms near one, small biases and sinks."""
    gen, short = _generator(seed, name), name.split(".")[-1]
    uniform = lambda: torch.rand(ps.shape, generator=gen, device=DEV)
    normal = lambda std: torch.randn(ps.shape, generator=gen, device=DEV) * std
    if short == "A_log":
        t = (uniform() * 15 + 1).log()
    elif short == "dt_bias":
        t = torch.expm1((uniform() * math.log(100.0) + math.log(0.001)).exp()).log()
    elif short.endswith("conv"):
        t = normal(0.4)
    elif ps.init == "ones":
        t = 1 + normal(0.1)
    elif ps.init == "zeros":
        t = normal(0.3)
    else:
        t = normal(0.02)
    return t.to(torch.float32 if ps.keep_float32 else dtype)


def _layer(kind):
    config, layer, place, sub = KINDS[kind]
    arch, cfg = parse_config(preset(config))
    spec = arch.model_spec(cfg)
    if place is None:
        return spec.layers[layer], dict(spec.layers[layer].parts["mixer"].params)
    part = spec.layers[layer].parts[place]
    return (part, dict(part.params)) if sub is None else (part.params["mixers"][sub],) + (dict(part.params["mixers"][sub].params),)


def _build(case, seed):
    """The part (or block) and its tensors by name."""
    kind, dtype = case["kind"], _dtype(case)
    spec, params = _layer(kind)
    if kind in ("block", "block_8b"):
        part, tensors = build_block(spec), {}
        for slot, sub in part.parts.items():
            mine = {n: _tensor("%s.%s" % (slot, n), ps, seed, dtype) for n, ps in sub.param_specs().items()}
            sub.load(mine)
            tensors.update({"%s.%s" % (slot, n): t for n, t in mine.items()})
        return part, tensors, params
    part = make_part(KINDS[kind][2], spec)
    tensors = {n: _tensor(n, ps, seed, dtype) for n, ps in part.param_specs().items()}
    part.load(tensors)
    return part, tensors, params


def _inputs(case, seed):
    """(part, tensors, parameters, step, normed rows, residual rows, cache, first state)."""
    part, tensors, params = _build(case, seed)
    gen, dtype = _generator(seed, "inputs"), _dtype(case)
    ctx, pages = _context(case, gen)
    hidden = params["hidden_size"]
    x = torch.randn(ctx.n_tokens, hidden, generator=gen, device=DEV).to(dtype)
    rows = torch.randn(ctx.n_tokens, hidden, generator=gen, device=DEV) * 0.02     # as token rows enter the first layer
    cache = first = None
    if case["kind"] in RECURRENT:
        shape = part.cache_request().shape
        state = torch.zeros((ctx.n_requests + 1,) + tuple(shape), device=DEV)
        if case["cached"]:
            state.normal_(0, 0.1, generator=gen)
            first = state.clone()
        cache = SlotStateCache(state)
    elif case["kind"] in PAGED:
        kv = part.cache_request()
        pool = lambda size: torch.randn(pages, kv.num_kv_heads, case["page"], size, generator=gen, device=DEV).to(dtype)
        cache = PagedKVCache(pool(kv.head_dim), pool(kv.value_dim), GROUP)
    return part, tensors, params, ctx, x, rows, cache, first


def _forward(s):
    part, ctx, cache = s["part"], s["ctx"], s["cache"]
    if s["kind"] in ("block", "block_8b"):
        stream = ResidualStream(s["rows"].clone(), s["dtype"])
        part.forward(stream, ctx, cache)
        return {"stream": stream.total(), "keys": cache.k, "values": cache.v}
    stream = ResidualStream(s["rows"].clone(), s["dtype"])
    if s["kind"] in RECURRENT:
        if s["empty"]:
            cache.state.zero_()          # a request's slot is cleared when it is admitted
        stream.add(part.forward(s["x"], ctx, cache))
        return {"stream": stream.total(), "state": cache.state[:ctx.n_requests]}
    if s["kind"] in PAGED:
        stream.add(part.forward(s["x"], ctx, cache))
        return {"stream": stream.total(), "keys": cache.k}
    stream.add(part.forward(s["x"], ctx))
    return {"stream": stream.total()}


def _whole():
    return {**preset(KINDS["whole"][0]), "num_hidden_layers": WHOLE_LAYERS}


def _prompt(case, seed, vocab):
    gen = torch.Generator().manual_seed(seed)
    return torch.randint(0, vocab, (case["tokens"],), generator=gen).tolist()


@torch.no_grad()
def prepare(case, seed):
    torch.backends.cuda.matmul.allow_tf32 = False
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    if case["kind"] == "whole":
        engine = Engine(config=_whole(), seed=seed, dtype=case["dtype"], page_size=case["page"], max_slots=2,
                        cache_tokens=case["tokens"] + 2 * case["page"], max_context=case["tokens"] + case["page"])
        expected = engine.model.expected_tensors()
        engine.model.load(lambda n: _tensor(n, expected[n], seed, _dtype(case)), _dtype(case))
        return {"kind": "whole", "engine": engine, "prompt": _prompt(case, seed, engine.vocab_size)}
    part, _, _, ctx, x, rows, cache, first = _inputs(case, seed)
    s = {"kind": case["kind"], "part": part, "ctx": ctx, "x": x, "rows": rows, "cache": cache, "dtype": _dtype(case), "graph": None,
         "empty": case["kind"] in RECURRENT and not case["cached"]}
    if _decode(case):
        # the layer's launches are recorded once, as the engine records a decode step, and replayed on each pass
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _forward(s)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["out"] = _forward(s)
        if first is not None:
            cache.state.copy_(first)
        s["graph"] = graph
    return s


@torch.no_grad()
def run(s):
    if s["kind"] == "whole":
        engine = s["engine"]
        engine.add_request("prompt")
        logits = engine.step([StepEntry("prompt", s["prompt"], [len(s["prompt"]) - 1])])
        engine.finish_request("prompt")
        return {"logits": logits}
    if s["graph"] is not None:
        s["graph"].replay()
        return s["out"]
    return _forward(s)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def _pairs(case, reach):
    """Visible (query, key) pairs, and cached keys that have to be read."""
    pairs = keys = 0
    for q, b in zip(*_lens(case)):
        seen = lambda p: min(p + 1, reach) if reach else p + 1
        pairs += sum(seen(b + t) for t in range(q))
        keys += min(b + q, (reach or b + q) + q)
    return pairs, keys


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    n = sum(_lens(case)[0])
    kind = case["kind"]
    if kind == "whole":
        c = _whole()
        h, f, d, layers = c["hidden_size"], c["intermediate_size"], c["head_dim"], c["num_hidden_layers"]
        per = h * d * (2 * c["num_attention_heads"] + 2 * c["num_key_value_heads"]) + 3 * h * f
        pairs = _pairs(case, None)[0]
        return {"bytes": size * (layers * per + c["vocab_size"] * h),
                "flops": 2.0 * layers * per * n + 2.0 * c["vocab_size"] * h + layers * 4.0 * c["num_attention_heads"] * d * pairs}
    p = _layer(kind)[1]
    h = p["hidden_size"]
    move = n * h * (size + 8)                                   # the input's rows, the stream's read and written
    if kind in ("block", "block_8b"):
        c = preset(KINDS[kind][0])
        weights = h * p["head_dim"] * (2 * p["num_heads"] + 2 * p["num_kv_heads"]) + 3 * h * c["intermediate_size"]
        pairs, keys = _pairs(case, None)
        return {"bytes": size * (weights + 2 * keys * p["num_kv_heads"] * p["head_dim"]) + move,
                "flops": 2.0 * weights * n + 4.0 * p["num_heads"] * p["head_dim"] * pairs}
    if kind.startswith("attention"):
        e = p["num_heads"] * p["head_dim"]
        weights = h * (e * (3 if p.get("gate") else 2) + 2 * p["num_kv_heads"] * p["head_dim"])
        pairs, keys = _pairs(case, p.get("window") or p.get("chunk"))
        return {"bytes": size * (weights + 2 * keys * p["num_kv_heads"] * p["head_dim"]) + move,
                "flops": 2.0 * weights * n + 4.0 * e * pairs}
    if kind.startswith("latent"):
        nh, d, rot, e, r = p["num_heads"], p["head_dim"], p["rot_dim"], p["v_head_dim"], p["kv_rank"]
        q_in = p.get("q_rank") or h
        weights = nh * (d + rot) * q_in + h * (r + rot) + nh * (d + e) * r + nh * e * h
        weights += (h * p["q_rank"] if p.get("q_rank") else 0) + (nh * e * h if p.get("gate") else 0)
        pairs, keys = _pairs(case, p.get("window"))
        return {"bytes": size * (weights + keys * (r + rot)) + move, "flops": 2.0 * weights * n + 2.0 * nh * (2 * r + rot) * pairs}
    if kind in RECURRENT:
        if kind == "state_space":
            inner, state = p["heads"] * p["vdim"], p["heads"] * p["vdim"] * p["state"]
            weights = h * (3 * inner + 2 * p["groups"] * p["state"])
        else:
            dim, vdim = p["dim"], p.get("vdim", p["dim"])
            inner, state = p["heads"] * vdim, p["heads"] * dim * vdim
            weights = h * (3 * inner + 2 * p.get("kv_heads", p["heads"]) * dim + (inner if kind == "general_delta" else 0))
        return {"bytes": size * weights + move + 4.0 * state * case["requests"] * (2 if case["cached"] else 1),
                "flops": 2.0 * weights * n + 6.0 * state * n}
    inner, per = p["expert_size"], 3 if p.get("gated") else 2
    touched = p["experts"] * (1 - (1 - p["top"] / p["experts"]) ** n)
    shared = per * h * (p.get("shared_size") or 0)
    return {"bytes": size * (per * h * inner * touched + shared) + 4 * h * p["experts"] + move,
            "flops": 2.0 * n * (per * h * inner * p["top"] + shared + h * p["experts"])}


def tolerance(case):
    """What the data types give.  bfloat16: a layer rounds its inner rows several times (measured against 64 bits: 2e-3 to
    4e-3 of the result); two correct orders of sums flip such roundings here and there.  Several layers carry them on
    (1e-2).  float32: sums of a few thousand terms, and accurate functions (1e-6)."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-3}
    if case["kind"] == "whole":
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 1e-2, "max": 0.3}


# ---- the layers in 64 bits ---------------------------------------------------------------------------------------------

def _rms(x, w, eps):
    x = x / (x.square().mean(-1, keepdim=True) + eps).sqrt()
    return x if w is None else x * w.double()


def _mm(x, w):
    return x @ w.double().t()


def _frequencies(dims, theta, scaling):
    """(frequency of each pair, factor on cosine and sine)."""
    f = [float(theta) ** (-2.0 * i / dims) for i in range(dims // 2)]
    if scaling is None:
        return f, 1.0
    if "low_freq_factor" in scaling:
        out = []
        for v in f:
            s = (scaling["original_max_position_embeddings"] * v / (2 * math.pi) - scaling["low_freq_factor"]) / (
                scaling["high_freq_factor"] - scaling["low_freq_factor"])
            s = min(max(s, 0.0), 1.0)
            out.append((1 - s) * v / scaling["factor"] + s * v)
        return out, 1.0
    pair = lambda turns: dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(theta))
    lo, hi = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [v / scaling["factor"] * r + v * (1 - r) for v, r in zip(f, ramp)], 0.1 * math.log(scaling["factor"]) + 1.0


def _turn(x, pos, dims, theta, scaling=None, interleaved=False):
    """x [n, heads, size] with its first ``dims`` sizes turned by the positions."""
    f, magnitude = _frequencies(dims, theta, scaling)
    angle = pos.double()[:, None, None] * torch.tensor(f, dtype=torch.float64, device=x.device)
    c, s = angle.cos() * magnitude, angle.sin() * magnitude
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if interleaved else (x[..., :dims // 2], x[..., dims // 2:dims])
    y = x.clone()
    if interleaved:
        y[..., 0:dims:2], y[..., 1:dims:2] = a * c - b * s, b * c + a * s
    else:
        y[..., :dims // 2], y[..., dims // 2:dims] = a * c - b * s, b * c + a * s
    return y


def _held(pool, table, count, page):
    """The first ``count`` cached rows of a request [count, heads, size]."""
    pages = table[:-(-count // page)].long() if count else table[:0].long()
    return pool[pages].double().permute(0, 2, 1, 3).flatten(0, 1)[:count]


def _attend(q, k, v, before, scale, window=None, chunk=None, sink=None, slopes=None):
    """q [n, heads, d] at positions before, before + 1, ...; k, v [before + n, kv heads, .]."""
    n, heads, dev = q.shape[0], q.shape[1], q.device
    pq, pk = torch.arange(before, before + n, device=dev)[:, None], torch.arange(k.shape[0], device=dev)[None, :]
    seen = pk <= pq
    if window:
        seen &= pk > pq - window
    if chunk:
        seen &= pk >= pq // chunk * chunk
    out = torch.empty(n, heads, v.shape[2], dtype=torch.float64, device=dev)
    for h in range(heads):
        g = h // (heads // k.shape[1])
        s = q[:, h] @ k[:, g].t() * scale
        if slopes is not None:
            s = s - slopes[h] * (pq - pk)
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(n, 1)], dim=1)
        w = s.softmax(-1)
        out[:, h] = (w[:, :-1] if sink is not None else w) @ v[:, g]
    return out


def _per_request(case, ctx):
    for i, (q, b) in enumerate(zip(*_lens(case))):
        at = ctx.host.q_start[i]
        yield i, slice(at, at + q), b


def _exact_general(case, t, p, ctx, x, cache):
    nh, g, d = p["num_heads"], p["num_kv_heads"], p["head_dim"]
    bias = lambda n: t[n].double() if n in t else 0.0
    n, pos = x.shape[0], ctx.positions
    q, k = (_mm(x, t[a + "_proj"]) + bias(a + "_bias") for a in "qk")
    v = (_mm(x, t["v_proj"]) + bias("v_bias")).view(n, g, d)
    q, k = q.view(n, nh, d), k.view(n, g, d)
    if p.get("qk_norm_eps") is not None:
        q, k = _rms(q, t["q_norm"], p["qk_norm_eps"]), _rms(k, t["k_norm"], p["qk_norm_eps"])
    if p.get("rotary"):
        r = p["rotary"]
        q, k = (_turn(u, pos, r["dims"], r["theta"], r.get("scaling"), r.get("layout") == "interleaved") for u in (q, k))
    if p.get("q_temperature"):
        c = p["q_temperature"]
        q = q * (1 + c["coef"] * (torch.floor((pos.double() + 1) / c["every"]) + 1).log())[:, None, None]
    y = torch.empty(n, nh, d, dtype=torch.float64, device=x.device)
    for i, rows, b in _per_request(case, ctx):
        table = ctx.block_tables[GROUP][i]
        keys = torch.cat([_held(cache.k, table, b, case["page"]), k[rows]])
        values = torch.cat([_held(cache.v, table, b, case["page"]), v[rows]])
        y[rows] = _attend(q[rows], keys, values, b, p["scale"], p.get("window"), p.get("chunk"), t.get("sink"), p.get("distance_slopes"))
    y = y.flatten(1)
    if p.get("gate"):
        y = y * _mm(x, t["g_proj"]).sigmoid()
    return _mm(y, t["o_proj"]) + bias("o_bias")


def _exact_latent(case, t, p, ctx, x, cache):
    nh, d, rot, e, r, eps = p["num_heads"], p["head_dim"], p["rot_dim"], p["v_head_dim"], p["kv_rank"], p["norm_eps"]
    n, pos, ro = x.shape[0], ctx.positions, p["rotary"]
    q = _mm(_rms(_mm(x, t["dq_proj"]), t["dq_norm"], eps) if p.get("q_rank") else x, t["q_proj"]).view(n, nh, d + rot)
    kv = _mm(x, t["dkv_proj"])
    turn = lambda u: _turn(u, pos, ro["head_dim"], ro["theta"], ro.get("scaling"), ro.get("layout") == "interleaved")
    q = torch.cat([q[..., :d], turn(q[..., d:])], -1)
    new = torch.cat([_rms(kv[:, :r], t["dkv_norm"], eps), turn(kv[:, None, r:])[:, 0]], -1)
    uk, uv = t["uk_proj"].double().view(nh, d, r), t["uv_proj"].double().view(nh, e, r)
    y = torch.empty(n, nh, e, dtype=torch.float64, device=x.device)
    for i, rows, b in _per_request(case, ctx):
        held = torch.cat([_held(cache.k, ctx.block_tables[GROUP][i], b, case["page"])[:, 0], new[rows]])
        c, kr = held[:, :r], held[:, r:]
        keys = torch.cat([torch.einsum("kr,hdr->khd", c, uk), kr[:, None].expand(-1, nh, -1)], -1)
        y[rows] = _attend(q[rows], keys, torch.einsum("kr,her->khe", c, uv), b, p["scale"], p.get("window"), None, t.get("sink"))
    y = y.flatten(1)
    if p.get("gate"):
        y = y * _mm(x, t["g_proj"]).sigmoid()
    return _mm(y, t["o_proj"])


def _silu(x):
    return x * x.sigmoid()


def _convolve(raw, w, tail, bias=None):
    """silu of the causal convolution of raw [n, c] behind the last inputs ``tail`` [c, taps - 1]; the new tail."""
    keep = w.shape[1] - 1
    full = torch.cat([tail.t(), raw])
    y = sum(full[j:j + raw.shape[0]] * w[:, j].double() for j in range(keep + 1))
    return _silu(y + (bias.double() if bias is not None else 0)), full[full.shape[0] - keep:].t()


def _walk(S, q, k, v, decay, beta=None, unit=None, removal=None, step=None):
    """The recurrence token by token: S [heads, dim, vdim]; q, k [n, heads, dim]; v [n, heads, vdim]; decay [n, heads, 1 or dim]."""
    out = torch.empty(v.shape, dtype=torch.float64, device=v.device)
    for i in range(v.shape[0]):
        if unit is not None:
            dot = torch.einsum("hd,hdv->hv", unit[i], S)
            S = S * decay[i][..., None] - removal[i][..., None] * dot[:, None] + k[i][..., None] * v[i][:, None]
        else:
            S = S * decay[i][..., None]
            u = v[i] if step is None else v[i] * step[i][:, None]
            if beta is not None:
                u = beta[i][:, None] * (v[i] - torch.einsum("hd,hdv->hv", k[i], S))
            S = S + k[i][..., None] * u[:, None]
        out[i] = torch.einsum("hd,hdv->hv", q[i], S)
    return out, S


def _exact_recurrent(case, t, p, ctx, x, first):
    kind, n = case["kind"], x.shape[0]
    h = p["heads"]
    dim = p["state"] if kind == "state_space" else p["dim"]
    vd, g = p.get("vdim", dim), p.get("kv_heads", p.get("groups", h))
    sp = torch.nn.functional.softplus
    heads = lambda u, m: u.reshape(n, m, -1)
    channels = taps = 0
    step = beta = unit = removal = None
    if kind in ("retention", "lightning"):
        q, k, v = heads(_mm(x, t["q_proj"]), h), heads(_mm(x, t["k_proj"]), h), heads(_mm(x, t["v_proj"]), h)
        if p.get("activation") == "silu":
            q, k, v = _silu(q), _silu(k), _silu(v)
        elif p.get("rotary"):
            ro = p["rotary"]
            q, k = (_turn(u, ctx.positions, ro["dims"], ro["theta"]) for u in (q, k))
            k = k * dim ** -0.5
        decay = torch.tensor(p["decay"], dtype=torch.float64, device=x.device).expand(n, h)[..., None]
    elif kind == "general_delta":
        q, k, v = (heads(_mm(x, t[a + "_proj"]), h) for a in "rkv")
        low = _mm(_mm(x, t["w1_proj"]).tanh(), t["w2_proj"]) + t["w_bias"].double()
        decay = heads((-p["decay_rate"] * low.sigmoid()).exp(), h)
        unit = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
        removal = unit * heads((_mm(x, t["a_proj"]) + t["a_bias"].double()).sigmoid(), h)
    elif kind == "state_space":
        z = _mm(x, t["in_proj"])
        inner, width = h * vd, h * vd + 2 * g * dim
        raw, conv_w, conv_b, channels, taps = z[:, inner:inner + width], t["conv"], t["conv_bias"], width, p["conv"]
        step = sp(z[:, inner + width:] + t["dt_bias"].double())
        decay = (-t["A_log"].double().exp() * step).exp()[..., None]
    else:
        raw = torch.cat([_mm(x, t[a + "_proj"]) for a in "qkv"], 1)
        conv_w, conv_b, channels, taps = torch.cat([t[a + "_conv"] for a in "qkv"]), None, raw.shape[1], p["conv"]
        beta = _mm(x, t["b_proj"]).sigmoid()
        a = _mm(x, t["a_proj"]) if p["decay"] == "head" else _mm(_mm(x, t["a1_proj"]), t["a2_proj"])
        rate = t["A_log"].double().exp()
        decay = (-rate[None, :, None] * heads(sp(a + t["dt_bias"].double()), h)).exp()
    out = torch.empty(n, h, vd, dtype=torch.float64, device=x.device)
    padded = -(-dim // 4) * 4
    total = -(-(h * vd * padded + channels * max(taps - 1, 0)) // 4) * 4
    state = torch.zeros(ctx.n_requests, total, dtype=torch.float64, device=x.device) if first is None else first[:ctx.n_requests].double()
    for i, rows, b in _per_request(case, ctx):
        S = state[i, :h * vd * padded].view(h, vd, padded)[..., :dim].transpose(1, 2)
        if channels:
            tail = state[i, h * vd * padded:h * vd * padded + channels * (taps - 1)].view(channels, taps - 1)
            y, new = _convolve(raw[rows], conv_w, tail, conv_b)
            tail.copy_(new)
            m = y.shape[0]
            if kind == "state_space":
                v, k, q = y[:, :h * vd].view(m, h, vd), y[:, h * vd:h * vd + g * dim], y[:, h * vd + g * dim:]
            else:
                q, k, v = y[:, :g * dim], y[:, g * dim:2 * g * dim], y[:, 2 * g * dim:].view(m, h, vd)
            q, k = q.view(m, g, dim), k.view(m, g, dim)
            if kind != "state_space":
                q, k = (u / (u.square().sum(-1, keepdim=True) + 1e-6).sqrt() for u in (q, k))
                q = q * dim ** -0.5
            qi, ki, vi = q.repeat_interleave(h // g, 1), k.repeat_interleave(h // g, 1), v
        else:
            qi, ki, vi = q[rows], k[rows], v[rows]
        pick = lambda u: None if u is None else u[rows]
        o, S = _walk(S, qi, ki, vi, decay[rows], pick(beta), pick(unit), pick(removal), pick(step))
        if kind == "state_space":
            o = o + t["D"].double()[None, :, None] * vi
        out[rows] = o
        state[i, :h * vd * padded].view(h, vd, padded)[..., :dim].copy_(S.transpose(1, 2))
    if kind == "state_space":
        y = (out.flatten(1) * _silu(z[:, :h * vd])).view(n, p["norm_groups"], -1)
        y = _rms(y, None, p["eps"]).flatten(1) * t["norm"].double()
    elif kind == "lightning":
        y = _rms(out.flatten(1), t["norm"], p["eps"]) * _mm(x, t["g_proj"]).sigmoid()
    elif kind == "retention":
        y = _rms(out, None, p["eps"]).flatten(1) * _silu(_mm(x, t["g_proj"]))
    elif kind == "general_delta":
        y = _rms(out, None, p["eps"]).flatten(1) * t["norm"].double() * _mm(x, t["g_proj"]).sigmoid()
    else:
        gate = _silu(_mm(x, t["g_proj"])) if p["gate"] == "silu" else _mm(_mm(x, t["g1_proj"]), t["g2_proj"]).sigmoid()
        y = _rms(out, t["norm"], p["eps"]).flatten(1) * gate
    return _mm(y, t["o_proj"]), state


def _exact_experts(t, p, x):
    s = _mm(x, t["router"]).softmax(-1)
    best, ids = s.topk(p["top"], dim=-1)
    weight = best if p.get("renorm", True) is False else best / (best.sum(-1, keepdim=True) + p.get("renorm_eps", 1e-20))
    weight = weight * p.get("route_scale", 1.0)
    act = _silu if p.get("gated") else (lambda u: u.relu().square())
    y = torch.zeros_like(x)
    for e in range(p["experts"]):
        at, slot = (ids == e).nonzero(as_tuple=True)
        if at.numel():
            inner = _mm(x[at], t["expert_%d_up" % e])
            inner = act(_mm(x[at], t["expert_%d_gate" % e])) * inner if p.get("gated") else act(inner)
            y.index_add_(0, at, _mm(inner, t["expert_%d_down" % e]) * weight[at, slot][:, None])
    if p.get("shared_size"):
        y = y + _mm(act(_mm(x, t["shared_up"])), t["shared_down"])
    return y


def _exact_block(x, c, t, pos, ranges):
    """A decoder layer over the rows x; ``ranges``: (rows, tokens before, cached keys, cached values) of every request."""
    nh, g, d, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
    n, h = x.shape[0], _rms(x, t["norm_1.weight"], eps)
    q, k, v = (_mm(h, t["mixer.%s_proj" % a]).view(n, -1, d) for a in "qkv")
    q, k = (_turn(u, pos, d, c["rope_theta"], c["rope_scaling"]) for u in (q, k))
    y = torch.empty(n, nh, d, dtype=torch.float64, device=x.device)
    for rows, b, ck, cv in ranges:
        y[rows] = _attend(q[rows], torch.cat([ck, k[rows]]), torch.cat([cv, v[rows]]), b, d ** -0.5)
    x = x + _mm(y.flatten(1), t["mixer.o_proj"])
    h = _rms(x, t["norm_2.weight"], eps)
    return x + _mm(_silu(_mm(h, t["feed_forward.gate_proj"])) * _mm(h, t["feed_forward.up_proj"]), t["feed_forward.down_proj"])


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "whole":
        return {"logits": _exact_whole(case, seed)}
    part, t, p, ctx, x, rows, cache, first = _inputs(case, seed)
    x, rows = x.double(), rows.double()
    if kind in ("block", "block_8b"):
        held = [(r, b, _held(cache.k, ctx.block_tables[GROUP][i], b, case["page"]), _held(cache.v, ctx.block_tables[GROUP][i], b, case["page"]))
                for i, r, b in _per_request(case, ctx)]
        return {"stream": _exact_block(rows, preset(KINDS[kind][0]), t, ctx.positions, held), "keys": None, "values": None}
    if kind in RECURRENT:
        y, state = _exact_recurrent(case, t, p, ctx, x, first)
        return {"stream": rows + y, "state": state}
    if kind in PAGED:
        y = (_exact_latent if kind.startswith("latent") else _exact_general)(case, t, p, ctx, x, cache)
        return {"stream": rows + y, "keys": None}
    return {"stream": rows + _exact_experts(t, p, x)}


def _exact_whole(case, seed):
    from yalis_b200.engine.model import Model
    c, dtype = _whole(), _dtype(case)
    arch, cfg = parse_config(c)
    spec = arch.model_spec(cfg)
    expected = Model(spec).expected_tensors()
    fetch = lambda n: _tensor(n, expected[n], seed, dtype)
    ids = torch.tensor(_prompt(case, seed, spec.vocab_size), device=DEV)
    pos, empty = torch.arange(len(ids), device=DEV), torch.zeros(0, c["num_key_value_heads"], c["head_dim"], dtype=torch.float64, device=DEV)
    table = fetch(spec.embedding_name)
    x = table[ids].double()
    for layer in spec.layers:
        t = {local: fetch(layer.weight_prefix + name) for local, name in layer.weight_names.items()}
        x = _exact_block(x, c, t, pos, [(slice(0, len(ids)), 0, empty, empty)])
    x = _rms(x[-1:], fetch(spec.final_norm_names["weight"]), c["rms_norm_eps"])
    return _mm(x, table if spec.head_name is None else fetch(spec.head_name))
