"""The exact attention of float32 heads of 64 and 128 in tiles of keys: every number of heads a key/value head, masks, caps, biases,
sinks and gates, contexts around a tile, against float64; however a request is cut and whatever runs beside it, the same bits."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
OPTIONS = [{}, {"window": 37}, {"chunk": 48}, {"window": 5, "chunk": 64, "softcap": 3.0, "sink": True, "gate": "value"},
           {"sink": "logits", "slopes": True, "gate": "head", "out_scale": 0.5}, {"rel": True, "window": 33}]


def plain(q, k, v, pos, o, scale):
    """One request in 64 bits: q [T, H, D], k and v [L, G, D]."""
    heads, length = q.shape[1], k.shape[0]
    k, v = (x.repeat_interleave(heads // k.shape[1], 1) for x in (k, v))
    s = torch.einsum("thd,lhd->thl", q, k) * scale
    j = torch.arange(length)
    back = pos[:, None] - j[None]
    if "slopes" in o:
        s = s - o["slopes"].double()[None, :, None] * back[:, None]
    if "rel" in o:
        s = s + o["rel"].double()[:, back.clamp(0, o["rel"].shape[1] - 1)].transpose(0, 1)
    if "softcap" in o:
        s = o["softcap"] * torch.tanh(s / o["softcap"])
    see = back >= 0
    see &= back < o.get("window", length + 1)
    if "chunk" in o:
        see &= j[None] >= pos[:, None] // o["chunk"] * o["chunk"]
    s = s.masked_fill(~see[:, None], -math.inf)
    if o.get("sink"):
        z = o["sink_logits"].double() if "sink_logits" in o else torch.zeros(heads).double()
        s = torch.cat([s, z[None, :, None].expand(s.shape[0], -1, 1)], -1)
        v = torch.cat([v, torch.zeros_like(v[:1])])
    y = torch.einsum("thl,lhd->thd", s.softmax(-1), v) * o.get("out_scale", 1.0)
    if "gate" in o:
        g = torch.sigmoid(o["gate"].double())
        y = y * (g[..., None] if g.shape[1] == heads else g.view_as(y))
    return y


@pytest.mark.parametrize("options", OPTIONS, ids=lambda o: "-".join(o) or "plain")
@pytest.mark.parametrize("heads,kv,dim", [(3, 3, 64), (4, 2, 128), (8, 2, 64), (6, 1, 128), (16, 2, 128), (8, 1, 64)])
def test_against_float64(heads, kv, dim, options):
    from yalis_b200.ops.attention import paged_attention_generic
    g = torch.Generator().manual_seed(heads * dim)
    rnd = lambda *s: torch.randn(*s, generator=g)
    lens, before, page = [1, 40, 7, 33, 2], [0, 0, 130, 31, 63], 16
    held = [a + b for a, b in zip(lens, before)]
    ks, vs = [rnd(h, kv, dim) for h in held], [rnd(h, kv, dim) for h in held]
    n = sum(lens)
    q = rnd(n, heads * dim)
    o = {k: v for k, v in options.items() if k in ("window", "chunk", "softcap", "out_scale")}
    extra = {}
    if options.get("sink"):
        extra["sink"] = True
        if options["sink"] == "logits":
            extra["sink_logits"] = rnd(heads)
    if "slopes" in options:
        extra["slopes"] = torch.rand(heads, generator=g) * 0.1
    if "rel" in options:
        extra["rel"] = rnd(heads, 20)
    gate = None
    if "gate" in options:
        gate = rnd(n, heads * dim if options["gate"] == "value" else heads)
    pages = sum(-(-h // page) for h in held) + 1
    pool_k, pool_v = torch.full((pages, kv, page, dim), math.inf), torch.full((pages, kv, page, dim), math.inf)
    order, table, at = torch.randperm(pages - 1, generator=g) + 1, torch.full((len(held), max(-(-h // page) for h in held)), -1, dtype=torch.int32), 0
    for r, h in enumerate(held):
        for i in range(-(-h // page)):
            table[r, i] = int(order[at])
            rows = slice(i * page, min(h, (i + 1) * page))
            pool_k[order[at], :, :rows.stop - rows.start] = ks[r][rows].transpose(0, 1)
            pool_v[order[at], :, :rows.stop - rows.start] = vs[r][rows].transpose(0, 1)
            at += 1
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    dev = lambda t: t.to(DEV) if torch.is_tensor(t) else t
    tokens = [(r, b + i) for r, (l, b) in enumerate(zip(lens, before)) for i in range(l)]

    def run(which):
        at = torch.tensor(which)
        return paged_attention_generic(q[at].to(DEV), pool_k.to(DEV), pool_v.to(DEV), ints([tokens[i][1] for i in which]),
                                       ints([tokens[i][0] for i in which]), table.to(DEV), heads, kv, dim, **o,
                                       gate=None if gate is None else gate[at].to(DEV), **{k: dev(v) for k, v in extra.items()}).cpu()

    got, a = run(list(range(n))), 0
    for r, l in enumerate(lens):
        mine = {**o, **extra, **({} if gate is None else {"gate": gate[a:a + l]})}
        want = plain(q[a:a + l].double().view(l, heads, dim), ks[r].double(), vs[r].double(), torch.arange(before[r], held[r]), mine, dim ** -0.5)
        # sums of up to 137 keys and 128 sizes, exponentials of differences of a few units: a few 2^-24 each
        assert (got[a:a + l].view_as(want).double() - want).norm() < 1e-6 * want.norm(), r
        a += l
    for which in (list(range(0, n, 2)), list(range(n))[::-1], list(range(3, 30)) + [0] + list(range(50, 60))):
        assert torch.equal(run(which), got[torch.tensor(which)])
    assert torch.equal(torch.cat([run([i]) for i in (0, 1, 9, 40, 41, n - 1)]), got[torch.tensor([0, 1, 9, 40, 41, n - 1])])


def test_later_values_and_missing_pages_do_not_reach_a_query():
    """An infinite value is seen by its own and later positions only; keys without a page count as masked."""
    from yalis_b200.ops.attention import paged_attention_generic
    g = torch.Generator().manual_seed(1)
    n, dim = 70, 64
    q, k, v = (torch.randn(n, dim, generator=g).to(DEV) for _ in range(3))
    pool_k, pool_v = k.new_zeros(5, 1, 16, dim), k.new_zeros(5, 1, 16, dim)
    pool_k.view(-1, dim)[:n], pool_v.view(-1, dim)[:n] = k, v
    args = lambda pv, t: (q, pool_k, pv, torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV),
                          torch.tensor([t], dtype=torch.int32, device=DEV), 1, 1, dim)
    whole = paged_attention_generic(*args(pool_v, [0, 1, 2, 3, 4]))
    bad = pool_v.clone()
    bad.view(-1, dim)[37] = math.inf
    got = paged_attention_generic(*args(bad, [0, 1, 2, 3, 4]))
    assert torch.equal(got[:37], whole[:37]) and bool(got[37:].isinf().all())
    got = paged_attention_generic(*args(pool_v, [0, 1, -1, 3, 9]))
    s = (q.double() @ k.double().t()) * dim ** -0.5
    j = torch.arange(n, device=DEV)
    s = s.masked_fill((j[None] > j[:, None]) | ((j[None] // 16 == 2) | (j[None] >= 64)), -math.inf)
    want = s.softmax(-1) @ v.double()
    assert (got.double() - want).norm() < 1e-6 * want.norm()


# heads and key/value heads that make a block take four heads and two queries, two and four, one and four in steps of these many tokens
FORMS = [(32, 8), (16, 8), (27, 9)]
LENS, BEFORE = [61, 1, 2, 47, 30, 3, 16], [0, 9, 30, 3, 101, 62, 32]


def step(heads, kv, dim, g, page=16):
    rnd = lambda *s: torch.randn(*s, generator=g)
    held = [a + b for a, b in zip(LENS, BEFORE)]
    ks, vs, q = [rnd(h, kv, dim) for h in held], [rnd(h, kv, dim) for h in held], rnd(sum(LENS), heads * dim)
    counts = [-(-h // page) for h in held]
    order, table, at = torch.randperm(sum(counts), generator=g) + 1, torch.full((len(held), max(counts)), -1, dtype=torch.int32), 0
    pools = [torch.full((sum(counts) + 1, kv, page, dim), math.nan) for _ in range(2)]
    for r, h in enumerate(held):
        for i in range(counts[r]):
            table[r, i] = int(order[at])
            rows = slice(i * page, min(h, (i + 1) * page))
            for pool, x in zip(pools, (ks, vs)):
                pool[order[at], :, :rows.stop - rows.start] = x[r][rows].transpose(0, 1)
            at += 1
    tokens = [(r, b + i) for r, (l, b) in enumerate(zip(LENS, BEFORE)) for i in range(l)]
    return q, ks, vs, pools, table, tokens


def attend(q, pools, table, tokens, heads, kv, dim, which, gate=None, **o):
    from yalis_b200.ops.attention import paged_attention_generic
    at = torch.tensor(which)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    dev = lambda t: t.to(DEV) if torch.is_tensor(t) else t
    return paged_attention_generic(q[at].to(DEV), pools[0].to(DEV), pools[1].to(DEV), ints([tokens[i][1] for i in which]), ints([tokens[i][0] for i in which]),
                                   table.to(DEV), heads, kv, dim, gate=None if gate is None else gate[at].to(DEV), **{k: dev(v) for k, v in o.items()}).cpu()


@pytest.mark.parametrize("options", OPTIONS, ids=lambda o: "-".join(o) or "plain")
@pytest.mark.parametrize("heads,kv", FORMS)
@pytest.mark.parametrize("dim", [64, 128])
def test_several_queries_a_block(heads, kv, dim, options):
    """Steps large enough for every form with several queries: portions that begin and end within a group of positions, single tokens beside
    them, against float64; the tokens one at a time, thus a query and a head a block, have the same bits."""
    g = torch.Generator().manual_seed(heads + dim)
    q, ks, vs, pools, table, tokens = step(heads, kv, dim, g)
    n = len(tokens)
    o = {k: v for k, v in options.items() if k in ("window", "chunk", "softcap", "out_scale")}
    gate = None if "gate" not in options else torch.randn(n, heads * dim if options["gate"] == "value" else heads, generator=g)
    if options.get("sink"):
        o["sink"] = True
        if options["sink"] == "logits":
            o["sink_logits"] = torch.randn(heads, generator=g)
    if "slopes" in options:
        o["slopes"] = torch.rand(heads, generator=g) * 0.1
    if "rel" in options:
        o["rel"] = torch.randn(heads, 20, generator=g)
    got, a = attend(q, pools, table, tokens, heads, kv, dim, list(range(n)), gate, **o), 0
    for r, l in enumerate(LENS):
        mine = {**o, **({} if gate is None else {"gate": gate[a:a + l]})}
        want = plain(q[a:a + l].double().view(l, heads, dim), ks[r].double(), vs[r].double(), torch.arange(BEFORE[r], BEFORE[r] + l), mine, dim ** -0.5)
        # as above
        assert (got[a:a + l].view_as(want).double() - want).norm() < 1e-6 * want.norm(), r
        a += l
    some = list(range(0, n, 9)) + [60, 61, 62, 63, 64, n - 1]
    alone = torch.cat([attend(q, pools, table, tokens, heads, kv, dim, [i], gate, **o) for i in some])
    assert torch.equal(alone, got[torch.tensor(some)])
    assert torch.equal(attend(q, pools, table, tokens, heads, kv, dim, list(range(n))[::-1], gate, **o), got.flip(0))


@pytest.mark.parametrize("heads,kv", FORMS)
@pytest.mark.parametrize("dim", [64, 128])
def test_several_queries_later_values_and_missing_pages(heads, kv, dim):
    g = torch.Generator().manual_seed(dim)
    q, ks, vs, pools, table, tokens = step(heads, kv, dim, g)
    every = list(range(len(tokens)))
    whole = attend(q, pools, table, tokens, heads, kv, dim, every)
    bad, place = [pools[0], pools[1].clone()], 37
    bad[1][table[0, place // 16], :, place % 16] = math.inf
    got = attend(q, bad, table, tokens, heads, kv, dim, every)
    reached = torch.tensor([r == 0 and p >= place for r, p in tokens])
    assert torch.equal(got[~reached], whole[~reached]) and bool(got[reached].isinf().all())
    gaps = table.clone()
    gaps[4, 2], gaps[0, 1] = -1, 10 ** 6                       # keys without a page count as masked
    got, a = attend(q, pools, gaps, tokens, heads, kv, dim, every), 0
    for r, l in enumerate(LENS):
        pos, j = torch.arange(BEFORE[r], BEFORE[r] + l), torch.arange(BEFORE[r] + l)
        k, v = (x[r].double().repeat_interleave(heads // kv, 1) for x in (ks, vs))
        s = torch.einsum("thd,lhd->thl", q[a:a + l].double().view(l, heads, dim), k) * dim ** -0.5
        gone = {4: 2, 0: 1}.get(r, -1)
        s = s.masked_fill(((j[None] > pos[:, None]) | (j[None] // 16 == gone))[:, None], -math.inf)
        want = torch.einsum("thl,lhd->thd", s.softmax(-1), v)
        assert (got[a:a + l].view_as(want).double() - want).norm() < 1e-6 * want.norm(), r
        a += l
