"""The recurrences' scan at the sizes where its split of a column changes, and portions around a group of four tokens and a
staged tile, against a float64 walk."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def walk(S, q, k, v, g, beta, unit, removal, selective, skip):
    out = []
    for t in range(v.shape[0]):
        if unit is not None:
            S = S * g[t][..., None] - removal[t][..., None] * torch.einsum("hd,hdv->hv", unit[t], S)[:, None] + k[t][..., None] * v[t][:, None]
        else:
            S = S * g[t][..., None]
            u = v[t] if beta is None else beta[t][:, None] * (v[t] if selective else v[t] - torch.einsum("hd,hdv->hv", k[t], S))
            S = S + k[t][..., None] * u[:, None]
        out.append(torch.einsum("hd,hdv->hv", q[t], S) + (skip[:, None] * v[t] if selective else 0))
    return torch.stack(out), S


@pytest.mark.parametrize("rule", ["constant", "token", "channel", "delta", "delta channel", "general", "selective"])
@pytest.mark.parametrize("dim,vdim", [(3, 5), (8, 64), (9, 33), (16, 1), (17, 70), (40, 8), (64, 16), (128, 128), (129, 17), (256, 9), (260, 31), (512, 6)])
def test_against_a_walk(rule, dim, vdim):
    from yalis_b200.ops.recurrent import StateLayout, state_scan
    g = torch.Generator().manual_seed(dim + vdim)
    heads, lens = 3, [1, 3, 4, 21, 0, 37]
    n, lay = sum(lens), StateLayout(heads, dim, vdim)
    rnd = lambda *s: torch.randn(*s, generator=g)
    q, k, v = rnd(n, heads, dim) / dim ** 0.5, rnd(n, heads, dim) / dim ** 0.5, rnd(n, heads, vdim)
    k = torch.nn.functional.normalize(k, dim=-1) if "delta" in rule or rule == "general" else k
    decay = {"constant": torch.rand(heads, generator=g)}.get(rule, 0.5 + 0.5 * torch.rand(n, heads, dim if "channel" in rule or rule == "general" else 1, generator=g))
    beta = torch.rand(n, heads, generator=g) if "delta" in rule or rule == "selective" else None
    unit = torch.nn.functional.normalize(rnd(n, heads, dim), dim=-1) if rule == "general" else None
    removal = unit * torch.rand(n, heads, 1, generator=g) if unit is not None else None
    skip = rnd(heads) if rule == "selective" else None
    rows = torch.zeros(len(lens) + 1, lay.total)
    rows[:-1] = rnd(len(lens), lay.total)
    state = rows[:, :lay.state_floats].view(-1, heads, vdim, lay.dim_padded)
    dev = lambda t: None if t is None else t.flatten(1).contiguous().to(DEV) if t.dim() > 1 else t.to(DEV)
    starts = torch.tensor([0] + lens).cumsum(0).to(torch.int32)

    def run(max_q_len, lo, hi, slot_rows, slots):
        cut = lambda t: None if t is None else dev(t[lo:hi]) if t.dim() > 1 else dev(t)
        return state_scan(cut(q), cut(k), cut(v), slot_rows, lay, slots[0], slots[1], kv_heads=heads, decay=cut(decay), beta=cut(beta),
                          unit=cut(unit), removal=cut(removal), max_q_len=max_q_len, selective=rule == "selective",
                          skip=dev(skip))

    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    got_rows = rows.to(DEV)
    got = run(max(lens), 0, n, got_rows, (starts.to(DEV), ints(list(range(len(lens)))))).cpu().view(n, heads, vdim)
    # the longest request again token by token: the same sums in the same order
    single_rows, at, single = rows.to(DEV), int(starts[5]), []
    for t in range(lens[5]):
        single.append(run(1, at + t, at + t + 1, single_rows, (ints([0, 1]), ints([5]))))
    assert torch.equal(torch.cat(single).cpu().view(-1, heads, vdim), got[at:])
    assert torch.equal(single_rows[5], got_rows[5])
    for i, l in enumerate(lens):
        a, b = int(starts[i]), int(starts[i]) + l
        cut = lambda t: None if t is None else t[a:b].double()
        d = decay.double().view(1, heads, 1).expand(l, heads, 1) if decay.dim() == 1 else cut(decay)
        first = state[i, :, :, :dim].double().transpose(1, 2)
        if l == 0:
            assert torch.equal(got_rows[i].cpu(), rows[i])
            continue
        want, S = walk(first, cut(q), cut(k), cut(v), d, cut(beta), cut(unit), cut(removal), rule == "selective",
                       None if skip is None else skip.double())
        # 32-bit sums of up to 512 terms carried over 37 tokens
        assert (got[a:b].double() - want).norm() < 2e-6 * want.norm()
        kept = got_rows[i, :lay.state_floats].cpu().view(heads, vdim, -1)[:, :, :dim].double().transpose(1, 2)
        assert (kept - S).norm() < 2e-6 * S.norm()


@pytest.mark.parametrize("dim,vdim", [(16, 40), (64, 128), (200, 33), (256, 128), (512, 6)])
@pytest.mark.parametrize("rule", ["delta", "general", "selective", "constant"])
def test_short_portions_have_a_tile_of_their_own(rule, dim, vdim):
    """Portions of at most four tokens give the bits of the longer tile, which the walk above is compared with."""
    from yalis_b200.ops.recurrent import StateLayout, state_scan
    g = torch.Generator(device=DEV).manual_seed(dim + vdim)
    heads, lens = 3, [2, 4, 1, 0, 3, 4]
    n, lay = sum(lens), StateLayout(heads, dim, vdim)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    unit = torch.nn.functional.normalize(rnd(n, heads, dim), dim=-1).flatten(1)
    more = {"delta": dict(decay=torch.rand(n, heads, generator=g, device=DEV), beta=torch.rand(n, heads, generator=g, device=DEV)),
            "general": dict(decay=torch.rand(n, heads * dim, generator=g, device=DEV), unit=unit, removal=0.5 * unit),
            "selective": dict(decay=torch.rand(n, heads, generator=g, device=DEV), beta=torch.rand(n, heads, generator=g, device=DEV),
                              selective=True, skip=rnd(heads)),
            "constant": dict(decay=torch.rand(heads, generator=g, device=DEV))}[rule]
    starts = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    rows, q, v = rnd(len(lens) + 1, lay.total), rnd(n, heads * dim) / dim ** 0.5, rnd(n, heads * vdim)
    got = []
    for longest in (4, 0):
        state = rows.clone()
        got.append((state_scan(q, unit, v, state, lay, starts, slots, kv_heads=heads, max_q_len=longest, **more), state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
