"""The plan of the routed rows: every entry has one slot among its expert's, tiles cover the slots, for entries that stay in registers and
ones that do not, many and few experts, entries of no expert."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("entries,experts,tile", [(1, 1, 16), (31, 3, 16), (4096, 16, 128), (8191, 33, 32), (8192, 1024, 128), (8193, 5, 16), (20000, 64, 128)])
def test_plan(entries, experts, tile):
    from yalis_b200.ops.experts import expert_plan
    g = torch.Generator().manual_seed(entries)
    ids = torch.randint(-1, experts + 1, (entries, 1), generator=g).to(torch.int32)
    plan = expert_plan(ids.to(DEV), experts, tile)
    flat = ids.flatten().long()
    flat[flat == experts] = -1                                  # an id past the last expert is no expert's either
    counts = torch.bincount(flat[flat >= 0], minlength=experts)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    used = int(offsets[-1])
    assert torch.equal(plan.offsets.cpu().long(), offsets)
    perm, inv = plan.perm.cpu()[:used].long(), plan.inv.cpu().flatten().long()
    assert torch.equal(perm.sort().values, (flat >= 0).nonzero().flatten())
    assert torch.equal(flat[perm], torch.repeat_interleave(torch.arange(experts), counts))
    assert torch.equal(inv[perm], torch.arange(used)) and bool((inv[flat < 0] == -1).all())
    want = [(e, int(offsets[e]) + t * tile) for e in range(experts) for t in range(-(-int(counts[e]) // tile))]
    n = int(plan.n_tiles.cpu())
    assert n == len(want)
    assert list(zip(plan.tile_expert.cpu()[:n].tolist(), plan.tile_slot.cpu()[:n].tolist())) == want
