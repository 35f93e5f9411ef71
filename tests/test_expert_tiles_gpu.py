"""Experts' products over tiles that end anywhere, and the router's rows taken two at a time, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bm", [64, 128, 256])
@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("width,inner", [(200, 72), (128, 520), (384, 1024)])
@pytest.mark.parametrize("most", [0, 5000])
def test_tiles_end_anywhere(bm, act, width, inner, most):
    """Experts with every number of slots around a tile's ``bm``, one with none; with ``most`` the average is large enough for
    two row blocks a tile, whose second one ends inside the expert's rows, past them, or past the tensor."""
    from yalis_b200.ops import experts as X
    counts = [1, 63, 64, 65, 0, 127, 129, 191, 192, 193, 255, 256, 257, 320, most, 5]
    g = torch.Generator().manual_seed(bm + width)
    ids = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    ids = ids[torch.randperm(ids.numel(), generator=g)].to(torch.int32)[:, None].cuda()
    n = ids.shape[0]
    x = torch.randn(n, inner, generator=g).bfloat16().cuda()
    w = (torch.randn(len(counts), width, inner, generator=g) / inner ** 0.5).bfloat16().cuda()
    plan = X.expert_plan(ids, len(counts), bm)
    rows = X.gather_rows(x, plan, 1)
    got = X.grouped_gemm_wstream(rows, w, plan, act=act).double()
    at = 0
    for e, c in enumerate(counts):
        want = rows[at:at + c].double() @ w[e].double().T
        # half a step of bfloat16, and float32 sums of `inner` terms; the square doubles the relative error
        slack = inner * 2.0 ** -23 * (rows[at:at + c].double().abs() @ w[e].double().abs().T)
        if act:
            want = want.clamp_min(0)
            slack = slack * (2 * want + slack)
            want = want * want
        assert bool(((got[at:at + c] - want).abs() <= 2.0 ** -8 * want.abs() + 1.01 * slack).all()), (e, c)
        at += c


def test_two_row_blocks_where_the_last_tile_is_half_empty():
    """Rows of an expert that end in the first block of their last tile: one block a tile for few of them, two for many."""
    from yalis_b200.ops import experts as X
    g = torch.Generator().manual_seed(7)
    ids = (torch.arange(1600) % 4).to(torch.int32)[:, None].cuda()
    x = torch.randn(1600, 72, generator=g).bfloat16().cuda()
    for width in (640, 2112):
        w = (torch.randn(4, width, 72, generator=g) / 72 ** 0.5).bfloat16().cuda()
        plan = X.expert_plan(ids, 4, 128)
        rows = X.gather_rows(x, plan, 1)
        got = X.grouped_gemm_wstream(rows, w, plan).double().view(4, 400, width)
        want = torch.einsum("esk,enk->esn", rows.double().view(4, 400, 72), w.double())
        size = torch.einsum("esk,enk->esn", rows.double().view(4, 400, 72).abs(), w.double().abs())
        # half a step of bfloat16, and float32 sums of 72 terms
        assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 72 * 2.0 ** -23 * size).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("experts", [1, 8, 9, 16, 17, 31])
@pytest.mark.parametrize("inner,side", [(256, True), (516, False), (130, True), (131, False)])
def test_router_rows(dtype, experts, inner, side):
    """1,027 tokens (blocks of eight, the last with three): a number of rows on either side of the warps, with and without
    the row of the gate, values of k that are loaded by four and one by one."""
    from yalis_b200.ops import experts as X
    g = torch.Generator().manual_seed(experts * 1000 + inner)
    x = torch.randn(1027, inner, generator=g).to(dtype).cuda()
    w = (torch.randn(experts, inner, generator=g) / inner ** 0.5).cuda()
    s = (torch.randn(inner, generator=g) / inner ** 0.5).cuda() if side else None
    out = X.route(x, w, experts, None, side=s)
    z = x.double() @ w.double().T
    slack = inner * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T).amax(1, keepdim=True)
    got = torch.zeros_like(z).scatter_(1, out[0].long(), out[1].double())
    want = torch.softmax(z, 1)
    # a logit's error twice (its own and the sum's), and a few roundings of the softmax itself
    assert bool(((got - want).abs() <= want * (2.1 * slack + 64 * 2.0 ** -23)).all())
    if side:
        zs = x.double() @ s.double()
        ss = inner * 2.0 ** -23 * (x.double().abs() @ s.double().abs())
        assert bool(((out[2].double() - torch.sigmoid(zs)).abs() <= torch.sigmoid(zs) * (1.1 * ss + 16 * 2.0 ** -23)).all())
    # one block a token gives the same bits: one order of sums
    few = X.route(x[:1000], w, experts, None, side=s)
    assert all(torch.equal(a[:1000], b) for a, b in zip(out, few))
