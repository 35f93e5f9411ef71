"""The activation with float32 results: rows of one group of four, of a block's share and just past it, columns of a wider matrix."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 4), (3, 3068), (2, 3072), (5, 3076), (2, 6148)])
def test_float32_results(dtype, rows, cols):
    from yalis_b200.ops.elementwise import activation
    g = torch.Generator().manual_seed(rows * cols)
    x = (3 * torch.randn(rows, cols + 8, generator=g)).to(DEV, dtype)[:, 4:4 + cols]
    got = activation(x, "silu", out_dtype=torch.float32)
    want = torch.nn.functional.silu(x.double())
    assert got.dtype == torch.float32 and got.shape == (rows, cols)
    # expf to 2 units in the last place, a sum, a division: below 8 units
    assert bool(((got.double() - want).abs() <= 8 * 2.0 ** -24 * want.abs() + 1e-37).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(512, 1024), (511, 1024), (600, 1020), (171, 3076), (86, 6148), (2100, 256), (16400, 16)])
def test_both_forms_have_the_same_bits(dtype, rows, cols):
    """A block a row for many wide rows, groups side by side otherwise: each row as in a call of its own."""
    from yalis_b200.ops.elementwise import activation
    g = torch.Generator().manual_seed(rows)
    x = (3 * torch.randn(rows, cols + 4, generator=g)).to(DEV, dtype)[:, 4:]
    got = activation(x, "silu", out_dtype=torch.float32)
    for r in (0, 1, rows // 2, rows - 1):
        assert torch.equal(got[r:r + 1], activation(x[r:r + 1], "silu", out_dtype=torch.float32))
    want = torch.nn.functional.silu(x.double())
    assert bool(((got.double() - want).abs() <= 8 * 2.0 ** -24 * want.abs() + 1e-37).all())      # as above
