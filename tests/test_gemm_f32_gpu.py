"""The float32 product in bfloat16 parts: edges of its tiles, K in parts of a step, both ways of reading rows, against float64 and
beside the product of FMAs; a row's result is the same bits whatever tile it falls into; infinities and very large and small values."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,k", [(128, 128), (129, 132), (300, 1000), (2048, 2048), (4100, 260), (130, 8192)])
def test_against_float64(n, k):
    from yalis_b200.ops.linear import gemm_f32, gemm_simt
    g = torch.Generator().manual_seed(n + k)
    for off, pad in ((0, 0), (4, 4), (1, 3)):                 # rows of a wider matrix; the last start off a 16-byte boundary
        x = torch.randn(700, k + pad + off, generator=g).to(DEV)[:, off:off + k]
        w = torch.randn(n, k + 8, generator=g).to(DEV)[:, 4:4 + k]
        whole = gemm_f32(x, w)
        want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
        assert bool(((whole.double() - want).abs() <= (k + 1) * 2.0 ** -24 * size).all())
        # no less exact than chains of FMAs, by more than chance allows for
        assert (whole.double() - want).norm() <= 1.02 * (gemm_simt(x, w).double() - want).norm()
        for m in (1, 15, 16, 17, 32, 33, 128, 129, 255, 256, 257, 513):
            assert torch.equal(gemm_f32(x[:m], w), whole[:m]), m
        low = x[:70].to(torch.bfloat16)
        assert torch.equal(gemm_f32(low, w, torch.float32), gemm_f32(low.float(), w))
        assert torch.equal(gemm_f32(x[:5], w, torch.bfloat16), whole[:5].to(torch.bfloat16))


def test_values_that_parts_cannot_hold():
    """Rows with infinities, NaN, the largest and the smallest values: what FMAs give; rows beside them keep their bits."""
    from yalis_b200.ops.linear import gemm_f32, gemm_simt
    g = torch.Generator().manual_seed(3)
    x, w = torch.randn(40, 260, generator=g).to(DEV), torch.randn(200, 260, generator=g).to(DEV)
    plain = gemm_f32(x, w)
    y = x.clone()
    y[1, 5], y[2, 7], y[3, 259], y[4], y[5] = float("inf"), float("nan"), 3.4e38, x[4] * 1e-36, 0.0
    y[6, 0], y[6, 1] = float("inf"), float("-inf")
    v = w.clone()
    v[9, 3], v[10, 2] = float("-inf"), 3.4e38
    got, want = gemm_f32(y, v), gemm_simt(y, v)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[want.isinf()], want[want.isinf()])
    # rows of tiny values: float32 FMAs in another order (the smallest products fall below the normal range)
    torch.testing.assert_close(got[4, :9], want[4, :9], rtol=1e-5, atol=1e-41)
    assert torch.equal(got[7:, :9], plain[7:, :9]) and torch.equal(got[0, 11:], plain[0, 11:])


@pytest.mark.parametrize("small,large", [(1e-37, 1e34), (1e-41, 1e20), (1e-42, 1e38), (1e-36, 1e30), (1e-30, 1e-14)])
@pytest.mark.parametrize("m", [5, 70, 300])
def test_small_values_beside_large_ones(small, large, m):
    """Values whose last parts bfloat16 does not hold, against values large enough to bring the product back: in rows of x, in rows of W, in
    single places; the rows beside them keep their bits."""
    from yalis_b200.ops.linear import gemm_f32
    g = torch.Generator().manual_seed(m)
    n, k = 140, 260
    x, w = torch.randn(m, k, generator=g).to(DEV), torch.randn(n, k, generator=g).to(DEV)
    plain = gemm_f32(x, w)
    y, v = x.clone(), w.clone()
    y[1] *= small
    v[7] *= large
    y[2] *= large
    v[9] *= small
    y[3], v[11] = 0.0, 0.0
    y[3, 5], v[11, 5], v[12, 5] = small, large, small
    y[4] = 0.0
    got = gemm_f32(y, v)
    want, size = y.double() @ v.double().t(), y.double().abs() @ v.double().abs().t()
    # float32 sums; below the normal numbers (products of two small values) a rounding is half of 1.4e-45
    bound = (k + 1) * (2.0 ** -24 * size + 1.4e-45)
    finite = size < 3e38                                       # (partial sums of FMAs may leave the range beyond)
    assert bool(((got.double() - want).abs() <= bound)[finite].all()), float(((got.double() - want).abs() / bound)[finite].max())
    assert not bool(got[4].any())
    others = torch.ones(n, dtype=torch.bool)
    others[[7, 9, 11, 12]] = False
    assert torch.equal(got[5:, others], plain[5:, others]) and torch.equal(got[0, others], plain[0, others])
