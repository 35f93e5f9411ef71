"""The float32 product at the edges of its tiles, aligned and not, against float64; a row's result is the same bits whatever
tile it falls into."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("k", [1, 15, 16, 63, 200])
@pytest.mark.parametrize("n", [1, 33, 130, 4100])
def test_tiles(n, k):
    from yalis_b200.ops.linear import gemm_simt
    g = torch.Generator().manual_seed(n + k)
    # rows of a wider matrix: strides that are not the width, and starts off a 16-byte boundary
    for pad, off in ((0, 0), (4, 4), (3, 1)):
        x = torch.randn(300, k + pad + off, generator=g).to(DEV)[:, off:off + k]
        w = torch.randn(n, k + pad + off, generator=g).to(DEV)[:, off:off + k]
        whole = gemm_simt(x, w)
        want = x.double() @ w.double().t()
        # a sum of k products, whatever its order: k 2^-24 of the sum of magnitudes at most
        assert bool(((whole.double() - want).abs() <= (k + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())).all())
        for m in (1, 31, 32, 33, 64, 65, 128, 129):
            assert torch.equal(gemm_simt(x[:m], w), whole[:m])
        assert torch.equal(gemm_simt(x[:70].to(torch.bfloat16), w, out_dtype=torch.float32),
                           gemm_simt(x[:70].to(torch.bfloat16).float(), w))


@pytest.mark.parametrize("rows", [65535 * 32, 65535 * 32 + 1, 65535 * 64])
def test_more_row_tiles_than_one_dimension_of_a_grid(rows):
    """Tiles of 32 rows, up to the most rows that are taken."""
    from yalis_b200.ops.linear import gemm_simt
    x = torch.arange(rows, device=DEV, dtype=torch.float32)[:, None] % 4099
    w = torch.tensor([[2.0], [-1.0], [0.5]], device=DEV)
    assert torch.equal(gemm_simt(x, w), x * w.t())


def test_rows_that_are_refused():
    from yalis_b200.ops._lib import KernelError
    from yalis_b200.ops.linear import gemm_simt
    with pytest.raises(KernelError):
        gemm_simt(torch.zeros(65535 * 64 + 1, 1, device=DEV), torch.ones(1, 1, device=DEV))
