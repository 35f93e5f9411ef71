"""The general decode attention deals its key tiles by the step: pairs in equal pieces, whole pairs, or all tiles evenly.  Every
way, and requests without a token between and behind the others, against plain attention in float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (heads, kv heads, size, cached tokens of each request, None: a request without a token)
STEPS = {
    "whole pairs, one a block": (16, 8, 64, [99] * 32),
    "whole pairs, two a block": (16, 8, 64, [199] * 64),
    "whole pairs, an odd number of them": (8, 8, 128, [70, 64, 10] * 25),
    "pieces of one long request": (16, 1, 128, [8000]),
    "pieces of which some pairs have fewer tiles": (4, 4, 64, [1900, 60, 1500]),
    "evenly, long beside short": (8, 4, 128, [9000] + [30] * 90),
    "evenly, more pairs than blocks": (16, 8, 64, [31 * i % 1500 for i in range(70)]),
    "none in between": (8, 4, 64, [300, None, 700, None, 5]),
    "none behind": (8, 4, 64, [300, 700, 64, 0, None, None, None, None]),
    "a single key": (2, 1, 256, [0]),
}


@pytest.mark.parametrize("step", STEPS)
def test_every_way_of_dealing(step):
    from yalis_b200.ops._lib import error_word
    from yalis_b200.ops.attention import decode_attention_general
    heads, kv, d, cached = STEPS[step]
    g = torch.Generator(device=DEV).manual_seed(len(step))
    page = 32
    per = [0 if c is None else c // page + 1 for c in cached]
    pages = sum(per) + 1
    pools = [torch.randn(pages, kv, page, d, generator=g, device=DEV).bfloat16() for _ in range(2)]
    order = torch.randperm(pages, generator=g, device=DEV)
    table = torch.full((len(cached), max(per)), -1, dtype=torch.int32, device=DEV)
    mine, at = [], 0
    for i, n in enumerate(per):
        mine.append(order[at:at + n])
        table[i, :n] = mine[-1].to(torch.int32)
        at += n
    live = [i for i, c in enumerate(cached) if c is not None]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    starts = [0]
    for c in cached:
        starts.append(starts[-1] + (c is not None))
    q = torch.randn(len(live), heads * d, generator=g, device=DEV).bfloat16()
    out = torch.full_like(q, float("nan"))
    counters = torch.zeros(len(cached) * kv, dtype=torch.int32, device=DEV)
    for _ in range(2):                                     # the counters are left as they were found
        out.fill_(float("nan"))
        decode_attention_general(q, pools[0], pools[1], ints([cached[i] for i in live]), ints(starts), table, heads, kv, d, d ** -0.5, out,
                                 counters=counters)
    assert int(error_word(DEV)) == 0 and not bool(counters.any())
    for row, i in enumerate(live):
        k, v = (p[mine[i]].double().permute(1, 0, 2, 3).flatten(1, 2)[:, :cached[i] + 1] for p in pools)
        mine_q = q[row].double().view(kv, heads // kv, d)
        want = torch.softmax(mine_q @ k.transpose(1, 2) * d ** -0.5, -1) @ v
        err = (out[row].double() - want.flatten()).abs()
        # the result's rounding to bfloat16 and the weights' to 16 bits
        assert bool((err <= 2.0 ** -8 * want.flatten().abs() + 3e-4 * want.abs().max()).all()), (i, float(err.max()))
