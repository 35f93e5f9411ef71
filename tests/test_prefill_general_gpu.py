"""The general forms of the tcgen05 prompt attention (tiles of 128 query rows and 64 keys) and of the decode attention that
deals tiles of 64 keys to a fixed grid, at the edges of their tiles, against plain attention in float64, option by option."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def plain(q, k, v, first, scale, window, chunk, softcap, sink, slopes):
    """q [n, h, d] at positions first ...; k, v [l, g, d]; float64."""
    n, h, l = q.shape[0], q.shape[1], k.shape[0]
    pos, key = torch.arange(first, first + n)[:, None], torch.arange(l)[None, :]
    hidden = key > pos
    if window:
        hidden |= key <= pos - window
    if chunk:
        hidden |= key < pos // chunk * chunk
    k, v = (t.repeat_interleave(h // k.shape[1], 1) for t in (k, v))
    s = torch.einsum("nhd,lhd->nhl", q, k) * scale
    if slopes is not None:
        s = s - slopes[None, :, None] * (pos - key)[:, None, :]
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    s = s.masked_fill(hidden[:, None, :], float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink[None, :, None].expand(n, -1, 1)], 2)
    return torch.einsum("nhl,lhd->nhd", s.softmax(-1)[:, :, :l], v)


# (head size, heads, kv heads, page, tokens brought, tokens held, options)
CASES = [
    (128, 16, 8, 64, [130, 65, 1], [0, 190, 127], dict(window=100)),
    (128, 6, 2, 16, [43, 129], [21, 64], dict(window=1, sink="learned")),
    (64, 4, 4, 8, [128, 17], [64, 250], dict(chunk=70, gate="element")),
    (64, 5, 1, 32, [26, 77], [0, 300], dict(chunk=64, sink="learned", gate="element", out_scale=0.7)),
    (128, 8, 4, 128, [65, 9], [63, 200], dict(softcap=5.0, sink="one")),
    (128, 3, 3, 64, [200], [57], dict(slopes=True, window=90, gate="head")),
    (64, 8, 2, 16, [33, 2], [100, 500], dict(slopes=True, softcap=3.0)),
    (128, 128, 1, 64, [3, 1], [300, 64], dict()),
]


# steps of single tokens
DECODE = [
    (128, 16, 8, 64, [0, 63, 64, 130, 2000], dict(window=100)),
    (128, 6, 2, 16, [21, 64, 300], dict(window=1, sink="learned")),
    (64, 4, 4, 8, [64, 250, 1], dict(chunk=70, gate="element")),
    (64, 16, 1, 32, [300, 7], dict(chunk=64, sink="learned", gate="element", out_scale=0.7)),
    (192, 8, 4, 64, [63, 200], dict(softcap=5.0, sink="one")),
    (256, 3, 3, 64, [57, 900, 3], dict(slopes=True, window=90, gate="head")),
    (128, 8, 2, 16, [100, 500] * 40, dict(slopes=True, softcap=3.0)),
    (128, 2, 2, 64, [4000], dict()),
]


@pytest.mark.parametrize("d,heads,kv,page,new,before,options", CASES + [(a, b, c, p, [1] * len(n), n, o) for a, b, c, p, n, o in DECODE])
def test_against_plain_attention(d, heads, kv, page, new, before, options):
    from yalis_b200.ops._lib import error_word
    from yalis_b200.ops.attention import decode_attention_general, prefill_attention_general
    g = torch.Generator().manual_seed(d + heads + page)
    window, chunk, scale = options.get("window"), options.get("chunk"), 0.9 / d ** 0.5
    sink = {"learned": torch.randn(heads, generator=g) * 2, "one": torch.zeros(heads)}.get(options.get("sink"))
    slopes = torch.rand(heads, generator=g) if options.get("slopes") else None
    held = [a + b for a, b in zip(new, before)]
    per = [-(-h // page) for h in held]
    pools = [torch.full((sum(per) + 3, kv, page, d), float("nan"), dtype=torch.bfloat16) for _ in range(2)]
    perm = torch.randperm(pools[0].shape[0], generator=g).tolist()
    table = torch.full((len(new), max(per)), -1, dtype=torch.int32)
    want, queries, pos, req, starts = [], [], [], [], [0]
    for i, (n, b) in enumerate(zip(new, before)):
        rows = [(torch.randn(held[i], kv, d, generator=g) * 1.5).to(torch.bfloat16) for _ in range(2)]
        least = max(b - window + 1 if window else 0, b // chunk * chunk if chunk else 0)
        for p in range(per[i]):
            if (p + 1) * page <= least:
                continue                                        # a page given back: no query sees its keys
            table[i, p] = perm.pop()
            for pool, r in zip(pools, rows):
                part = r[p * page:(p + 1) * page].transpose(0, 1)
                pool[table[i, p], :, :part.shape[1]] = part
        q = (torch.randn(n, heads, d, generator=g) * 1.5).to(torch.bfloat16)
        queries.append(q)
        want.append(plain(q.double(), rows[0].double(), rows[1].double(), b, scale, window, chunk, options.get("softcap"),
                          None if sink is None else sink.double(), None if slopes is None else slopes.double()))
        pos += range(b, b + n)
        req += [i] * n
        starts.append(starts[-1] + n)
    total = len(pos)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    wide = torch.full((total, heads * d + 24), float("nan"), dtype=torch.bfloat16, device=DEV)
    out = wide[:, 8:8 + heads * d]                              # a column block of a wider matrix
    gate = None
    if options.get("gate"):
        gate = torch.randn(total, heads * d if options["gate"] == "element" else heads, generator=g).to(torch.bfloat16)
    args = [torch.cat(queries).flatten(1).contiguous().to(DEV), pools[0].to(DEV), pools[1].to(DEV), ints(pos), ints(starts), table.to(DEV),
            max(new), heads, kv, d, scale, out]
    call = prefill_attention_general
    if max(new) == 1:
        call = decode_attention_general
        del args[6]
    call(*args, window=window, chunk=chunk, softcap=options.get("softcap"), sink=sink is not None,
         sink_logits=sink.to(DEV) if options.get("sink") == "learned" else None, slopes=None if slopes is None else slopes.to(DEV),
         gate=None if gate is None else gate.to(DEV), out_scale=options.get("out_scale", 1.0))
    assert int(error_word(DEV)) == 0
    want = torch.cat(want) * options.get("out_scale", 1.0)
    if gate is not None:
        want = want * gate.double().sigmoid().view(total, heads, -1)
    got = out.double().cpu().view(total, heads, d)
    # the result's rounding to bfloat16 (2^-9 of the element), the weights' to 16 bits and the scores' 32-bit sums
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 3e-4 * want.abs().max()).all()), float(((got - want).abs() / want.abs().max()).max())
    assert bool(wide[:, :8].isnan().all()) and bool(wide[:, 8 + heads * d:].isnan().all())
