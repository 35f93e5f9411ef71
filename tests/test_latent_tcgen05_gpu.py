"""The tcgen05 form of the latent attention at the edges of its tiles (128 query rows, 64 rows of the cache) against plain
attention in float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def plain(q, rows, r, scale, window, first, sink):
    """q [n, heads, w] at positions first, first + 1, ...; rows [l, w]; float64."""
    s = torch.einsum("nhw,lw->nhl", q, rows) * scale
    pos, key = torch.arange(first, first + q.shape[0])[:, None], torch.arange(rows.shape[0])[None, :]
    hidden = (key > pos) | ((key <= pos - window) if window else torch.zeros_like(key > pos))
    s = s.masked_fill(hidden[:, None, :], float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink[None, :, None].expand(q.shape[0], -1, 1)], dim=2)
    w = s.softmax(-1)[:, :, :rows.shape[0]]
    return torch.einsum("nhl,lr->nhr", w, rows[:, :r])


# (r, p, heads, page, window, sink, splits, tokens brought, tokens held before)
CASES = [
    (64, 64, 3, 8, None, False, 1, [1, 43, 129], [63, 0, 64]),
    (128, 0, 16, 16, 70, True, 1, [9, 8, 1], [0, 250, 127]),
    (256, 64, 16, 64, 100, False, 1, [130, 65], [0, 190]),
    (256, 64, 16, 64, 1, True, 1, [17], [60]),
    (256, 64, 24, 32, None, True, 16, [1, 1, 1], [1024, 0, 63]),
    (256, 64, 128, 128, None, False, 3, [1, 1], [200, 64]),
    (384, 64, 24, 64, None, True, 1, [33, 70], [100, 0]),
    (384, 64, 24, 128, 150, False, 5, [1, 1], [700, 128]),
]


@pytest.mark.parametrize("r,p,heads,page,window,sink,splits,new,before", CASES)
def test_against_plain_attention(r, p, heads, page, window, sink, splits, new, before):
    from yalis_b200.ops._lib import error_word, i32 as c_int, lib
    from yalis_b200.ops.latent import latent_attention_mma
    assert lib().yalis_latent_attention_tcgen05_supports(c_int(r), c_int(p), c_int(page))
    g = torch.Generator().manual_seed(r + heads + splits)
    w, scale = r + p, 0.4 / (r + p) ** 0.5
    held = [a + b for a, b in zip(new, before)]
    per = [-(-h // page) for h in held]
    pool = torch.full((sum(per) + 3, 1, page, w), float("nan"), dtype=torch.bfloat16)       # what no request wrote is NaN
    perm = torch.randperm(pool.shape[0], generator=g).tolist()
    table = torch.full((len(new), max(per)), -1, dtype=torch.int32)
    zs = torch.randn(heads, generator=g) * 2 if sink else None
    want, queries, pos, req, starts = [], [], [], [], [0]
    for i, (n, b) in enumerate(zip(new, before)):
        rows = (torch.randn(held[i], w, generator=g) * 2).to(torch.bfloat16)
        for t in range(held[i]):
            if window and t + page <= b - window + 1 and t % page == 0:
                perm.pop()                                                                # a page given back behind the window
            elif t % page == 0 or table[i, t // page] >= 0:
                if t % page == 0:
                    table[i, t // page] = perm.pop()
                pool[table[i, t // page], 0, t % page] = rows[t]
        q = (torch.randn(n, heads, w, generator=g) * 2).to(torch.bfloat16)
        queries.append(q)
        want.append(plain(q.double(), rows.double(), r, scale, window, b, None if zs is None else zs.double()))
        pos += range(b, b + n)
        req += [i] * n
        starts.append(starts[-1] + n)
    q = torch.cat(queries).to(DEV)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q_lat = q[:, :, :r].transpose(0, 1).contiguous()                                       # head-major, as the mixer gives it
    out = torch.full((heads, len(pos), r), float("nan"), dtype=torch.bfloat16, device=DEV)
    latent_attention_mma(q_lat.transpose(0, 1), q[:, :, r:].float().contiguous(), out.transpose(0, 1), pool.to(DEV), ints(pos),
                         ints(starts), ints(req), table.to(DEV), len(new), max(new), scale, window, n_splits=splits,
                         sink=None if zs is None else zs.to(DEV))
    assert int(error_word(DEV)) == 0
    got, want = out.transpose(0, 1).double().cpu(), torch.cat(want)
    # the result's rounding to bfloat16 (2^-9 of the element) and the weights' to 16 bits (2^-17 of the weighted sum of
    # magnitudes, below sqrt(keys) of the result's size here)
    err = (got - want).abs()
    assert bool((err <= 2.0 ** -8 * want.abs() + 2e-4 * want.abs().max()).all()), float((err / want.abs().max()).max())
