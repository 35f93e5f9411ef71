"""Element-wise kernels that take four values a thread where rows allow it: sizes and starts on both sides of that rule give
the results of the plain expression."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows,width", [(1, 1), (3, 7), (5, 4), (129, 12), (7, 1030)])
@pytest.mark.parametrize("parts", [0, 1, 3, 17])
def test_residual_add(rows, width, parts):
    from yalis_b200.ops.elementwise import residual_add
    g = torch.Generator().manual_seed(rows + width + parts)
    x = torch.randn(rows * width + 4, generator=g).to(DEV)
    for off in (0, 1):
        mine = x.clone()[off:off + rows * width].view(rows, width)
        want = mine.clone()
        if parts == 0:
            delta = torch.randn(rows, width, generator=g).to(torch.bfloat16).to(DEV)
            want += delta.float()
        else:
            delta = torch.randn(parts, rows, width, generator=g).to(DEV)
            for p in delta:
                want += p                              # in order: the same roundings
        residual_add(mine, delta)
        assert torch.equal(mine, want)


@pytest.mark.parametrize("heads,vdim", [(1, 4), (3, 5), (5, 128), (2, 132), (3, 512), (2, 516), (4, 64)])
@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_head_norm_gate(heads, vdim, kind, dtype):
    from yalis_b200.ops.recurrent import head_norm_gate
    g = torch.Generator().manual_seed(heads + vdim + kind)
    n, c = 5, heads * vdim
    o, z = torch.randn(n, c, generator=g), torch.randn(n, c + 8, generator=g).to(dtype)
    weight = torch.randn(c if kind == 2 else vdim, generator=g)
    req = torch.tensor([0, 0, -1, 1, 1], dtype=torch.int32, device=DEV)
    for off in (0, 1, 4):
        gate = z[:, off:off + c]
        out = torch.full((n, c + 8), 3.0, dtype=dtype, device=DEV)
        head_norm_gate(o.to(DEV), heads, vdim, 1e-5, req, out[:, off:off + c], weight=weight.to(DEV), gate=z.to(DEV)[:, off:off + c],
                       gate_kind=kind, out_scale=0.5)
        x = o.double().view(n, heads, vdim)
        x = x / (x.square().mean(-1, keepdim=True) + 1e-5).sqrt() * weight.double().view(-1, vdim)
        act = {0: torch.ones_like(gate.double()), 1: gate.double() * gate.double().sigmoid(), 2: gate.double().sigmoid()}[kind]
        want = x.flatten(1) * act * 0.5
        got = out[:, off:off + c].double().cpu()
        live = [0, 1, 3, 4]
        # 32-bit arithmetic of a dozen operations, then the output's rounding
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-6
        assert bool(((got - want).abs()[live] <= eps * want.abs()[live] + 1e-7).all())
        assert bool((out[2] == 3.0).all()) and bool((out[:, :off] == 3.0).all()) and bool((out[:, off + c:] == 3.0).all())


@pytest.mark.parametrize("heads,e", [(1, 4), (3, 6), (16, 128), (5, 20)])
@pytest.mark.parametrize("dtype,x_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_sigmoid_gate(heads, e, dtype, x_dtype):
    from yalis_b200.ops.latent import sigmoid_gate
    g = torch.Generator().manual_seed(heads + e)
    n = 7
    x = torch.randn(heads, n, e, generator=g).to(x_dtype)              # head-major, as the attention leaves it
    z = (torch.randn(n, heads * e + 8, generator=g) * 3).to(dtype)
    want_x = x.transpose(0, 1).flatten(1).double()
    for off in (0, 2, 4):
        out = torch.full((n, heads * e + 8), 3.0, dtype=dtype, device=DEV)
        sigmoid_gate(x.to(DEV).transpose(0, 1), z.to(DEV)[:, off:off + heads * e], out[:, off:off + heads * e])
        want = want_x * z[:, off:off + heads * e].double().sigmoid()
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6
        assert bool(((out[:, off:off + heads * e].double().cpu() - want).abs() <= eps * want.abs() + 1e-7).all())
        assert bool((out[:, :off] == 3.0).all()) and bool((out[:, off + heads * e:] == 3.0).all())
