"""A visible key whose page is not mapped is read as zeros, not from anywhere, and the error word says so; a page that no query
sees may be gone."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
I32 = dict(dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("missing", [-1, 1 << 20])
@pytest.mark.parametrize("at,window,flagged", [(2, None, True), (0, None, True), (0, 40, False), (1, 40, True)])
@pytest.mark.parametrize("tokens", [1, 20])
def test_general_forms(missing, at, window, flagged, tokens):
    from yalis_b200.ops._lib import FLAG_BAD_PAGE
    from yalis_b200.ops.attention import decode_attention_general, prefill_attention_general
    heads, kv, d, page, held = 4, 2, 64, 32, 90
    pool = torch.randn(8, kv, page, d, device=DEV).bfloat16()
    table = torch.tensor([[3, 1, 6]], **I32)
    table[0, at] = missing
    q = torch.randn(tokens, heads * d, device=DEV).bfloat16()
    pos, starts = torch.arange(held - tokens, held, **I32), torch.tensor([0, tokens], **I32)
    out, error = torch.empty_like(q), torch.zeros(1, **I32)
    if tokens == 1:
        decode_attention_general(q, pool, pool, pos, starts, table, heads, kv, d, 0.1, out, window=window, error_flag=error)
    else:
        # the first query stands at 70: with a window of 40 it sees keys from 31
        prefill_attention_general(q, pool, pool, pos, starts, table, tokens, heads, kv, d, 0.1, out, window=window, error_flag=error)
        flagged = True
    assert int(error) == (FLAG_BAD_PAGE if flagged else 0) and bool(out.isfinite().all())


@pytest.mark.parametrize("window,flagged", [(None, True), (40, False)])
def test_latent(window, flagged):
    from yalis_b200.ops._lib import FLAG_BAD_PAGE, error_word
    from yalis_b200.ops.latent import latent_attention_mma
    heads, r, p, page, held = 16, 128, 64, 32, 90
    pool = torch.randn(8, 1, page, r + p, device=DEV).bfloat16()
    table = torch.tensor([[-1, 1, 6]], **I32)
    q, rot = torch.randn(1, heads, r, device=DEV).bfloat16(), torch.randn(1, heads, p, device=DEV)
    out, word = torch.empty_like(q), error_word(DEV)
    assert int(word) == 0
    latent_attention_mma(q, rot, out, pool, torch.tensor([held - 1], **I32), torch.tensor([0, 1], **I32), torch.zeros(1, **I32), table, 1, 1,
                         0.1, window)
    found = int(word)
    word.zero_()
    assert found == (FLAG_BAD_PAGE if flagged else 0) and bool(out.isfinite().all())
