"""Heads that are normed one by one and turn, in registers: sizes around the lanes of a head, both layouts, against float64."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,vdim,rot", [(8, 8, 8), (64, 64, 16), (64, 128, 64), (72, 40, 24), (128, 128, 128), (128, 128, 64), (136, 128, 8),
                                          (256, 256, 248), (128, 64, 12), (128, 128, 0)])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("normed", [False, True])
@pytest.mark.parametrize("dtypes", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
def test_heads_turn(dim, vdim, rot, interleaved, normed, dtypes):
    from yalis_b200.ops.elementwise import qkv_prepare
    src_dtype, out_dtype = dtypes
    nq, nk, n = 7, 2, 600
    g = torch.Generator().manual_seed(dim * 1000 + rot)
    width = (nq + nk) * dim + nk * vdim
    src = torch.randn(n, width + 16, generator=g).to(src_dtype).cuda()[:, 8:8 + width + 8]
    src = src if src_dtype == torch.float32 else src.contiguous()
    offsets = (0, nq * dim, (nq + nk) * dim)
    sizes = (nq * dim, nk * dim, nk * vdim)
    biases = tuple(torch.randn(s, generator=g).to(src_dtype).cuda() for s in sizes) if dim != 64 else (None, None, None)
    norms = tuple((1 + 0.1 * torch.randn(dim, generator=g)).cuda() for _ in range(2)) if normed else (None, None)
    freq = (10000.0 ** (-torch.arange(0, rot, 2, dtype=torch.float32) / max(rot, 1))).cuda() if rot else None
    positions = torch.arange(n, dtype=torch.int32).cuda()
    req = torch.zeros(n, dtype=torch.int32).cuda()

    def run(rows):
        return qkv_prepare(src[:rows], offsets, nq, nk, dim, vdim, positions[:rows], req[:rows], out_dtype=out_dtype, biases=biases,
                           q_norm=norms[0], k_norm=norms[1], norm_eps=1e-6, inv_freq=freq, q_scale=0.5, k_scale=1.25,
                           interleaved=interleaved, rot_scale=1.1, q_temperature=(0.1, 64))

    got = run(n)
    pos = positions.double()
    angle = (pos[:, None].float() * freq).double() if rot else None
    for i, heads in enumerate((nq, nk, nk)):
        x = src[:, offsets[i]:offsets[i] + sizes[i]].double()
        if biases[i] is not None:
            x = x + biases[i].double()
        x = x.view(n, heads, -1)
        big = x.abs().amax(-1, keepdim=True)
        if i < 2:
            if normed:
                r = 1 / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)
                x, big = x * r * norms[i].double(), big * r * 1.6
            if rot:
                cs, sn = torch.cos(angle)[:, None] * 1.1, torch.sin(angle)[:, None] * 1.1
                t = x[..., :rot]
                a, b = (t[..., 0::2], t[..., 1::2]) if interleaved else (t[..., :rot // 2], t[..., rot // 2:])
                o = (a * cs - b * sn, b * cs + a * sn)
                o = torch.stack(o, -1).flatten(-2) if interleaved else torch.cat(o, -1)
                x = torch.cat((o, x[..., rot:]), -1)
            factor = torch.full_like(pos, 1.25) if i else 0.5 * (1 + 0.1 * torch.log(torch.floor((pos + 1) / 64) + 1))
            x, big = x * factor[:, None, None], big * factor[:, None, None]
        y = got[i].double().view(n, heads, -1)
        # float32 arithmetic: a sum of squares of up to 256 terms (its root halves the error) and some ten roundings
        slack = 2.2 * big * (256 + 24) * 2.0 ** -24 + (2.0 ** -8 * x.abs() if out_dtype == torch.bfloat16 else 0)
        assert bool(((y - x).abs() <= slack).all()), (i, ((y - x).abs() / slack).max().item())
    few = run(5)
    assert all(torch.equal(a[:5], b) for a, b in zip(got, few))


@pytest.mark.parametrize("dim", [64, 128, 256])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("dtypes", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
def test_steps_of_more_blocks_than_places_have_the_same_bits(dim, interleaved, dtypes):
    """The form in fewer registers, for many blocks, beside the other one."""
    from yalis_b200.ops.elementwise import qkv_prepare
    nq, nk, n, few = 7, 2, 2300, 310
    g = torch.Generator().manual_seed(dim)
    src = torch.randn(n, (nq + 2 * nk) * dim, generator=g).to(dtypes[0]).cuda()
    norm, freq = torch.rand(dim, generator=g).cuda(), torch.rand(dim // 2, generator=g).cuda()
    positions, req = torch.arange(n, dtype=torch.int32).cuda(), torch.zeros(n, dtype=torch.int32).cuda()

    def run(a, b):
        return qkv_prepare(src[a:b], (0, nq * dim, (nq + nk) * dim), nq, nk, dim, dim, positions[a:b].contiguous(), req[a:b].contiguous(),
                           out_dtype=dtypes[1], q_norm=norm, k_norm=norm, norm_eps=1e-6, inv_freq=freq, interleaved=interleaved)

    whole = run(0, n)
    for a in (0, 1100, n - few):
        for x, y in zip(run(a, a + few), whole):
            assert torch.equal(x, y[a:a + few])
