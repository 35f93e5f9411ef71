"""The short convolution of long steps, two tokens a warp: the same bits as token by token, over portions that begin, end and are shorter than
the taps within a tile, rows of no request, other taps, heads and types."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("channels,kv_heads,taps,per_channel,bias", [(512, 1, 4, False, False), (384, 1, 3, True, True), (1280, 0, 4, False, True),
                                                                    (128, 0, 2, False, False), (256, 1, 1, True, False)])
def test_same_bits_as_token_by_token(dtype, channels, kv_heads, taps, per_channel, bias):
    from yalis_b200.ops.recurrent import delta_prepare
    g = torch.Generator().manual_seed(channels + taps)
    lens, pad, heads = [1, 2, 3, 130, 5, 120, 7], 3, 2
    n = sum(lens) + pad                                         # the last rows belong to no request
    wide = torch.randn(n, channels + 5, generator=g).to(DEV, dtype)
    x = wide[:, 3:3 + channels]                                 # rows on odd boundaries
    w = torch.randn(channels, taps, generator=g).to(DEV)
    first = torch.randn(len(lens) + 1, channels * (taps - 1) + 4, generator=g).to(DEV)
    slots = torch.tensor([3, 0, 7, 1, 5, 2, 4], dtype=torch.int32, device=DEV)
    a_cols = heads * 128 if per_channel else heads
    a, b = torch.randn(n, a_cols, generator=g).to(DEV, dtype), torch.randn(n, heads, generator=g).to(DEV, dtype)
    rates = dict(a_log=torch.rand(heads, generator=g).to(DEV), dt_bias=torch.randn(a_cols, generator=g).to(DEV), unit_heads=kv_heads, dim=128,
                 q_scale=0.3, conv_bias=torch.randn(channels, generator=g).to(DEV) if bias else None)
    starts = torch.tensor([0] + lens).cumsum(0)
    req = torch.cat([torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)), torch.full((pad,), -1)]).to(torch.int32).to(DEV)
    rows = first.clone()
    got = delta_prepare(x, w, rows, 2, req, starts.to(torch.int32).to(DEV), slots, a_raw=a, b_raw=b, **rates)
    kept = first.clone()
    for r, l in enumerate(lens):
        for t in range(l):
            i = int(starts[r]) + t
            want = delta_prepare(x[i:i + 1], w, kept, 2, torch.zeros(1, dtype=torch.int32, device=DEV),
                                 torch.tensor([0, 1], dtype=torch.int32, device=DEV), slots[r:r + 1].contiguous(), a_raw=a[i:i + 1],
                                 b_raw=b[i:i + 1], single_tokens=True, **rates)
            for u, v in zip(got, want):
                assert torch.equal(u[i:i + 1], v), (r, t)
    assert torch.equal(rows, kept)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("channels,kv_heads,taps,per_channel,bias", [(4096, 16, 4, False, False), (3968, 3, 3, True, True), (4224, 0, 4, False, True),
                                                                    (3968, 0, 2, False, False), (4096, 1, 1, True, False)])
def test_as_many_values_as_take_tiles(dtype, channels, kv_heads, taps, per_channel, bias):
    """Steps of 271 tokens with 2^20 values and more."""
    test_same_bits_as_token_by_token(dtype, channels, kv_heads, taps, per_channel, bias)
