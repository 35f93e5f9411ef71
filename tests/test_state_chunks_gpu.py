"""The recurrences by chunks of sixteen tokens: portions around a chunk's end beside short ones, every rule that goes this way, column
tiles that are not full, against a float64 walk and beside the walk token by token."""

import pytest
import torch

from test_state_scan_gpu import walk

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
RULES = ["constant", "token", "delta constant", "delta", "selective"]


def inputs(rule, heads, kv_heads, vdim, lens, g, keep=0.5):
    n, dim = sum(lens), 128
    rnd = lambda *s: torch.randn(*s, generator=g)
    q, k, v = rnd(n, kv_heads, dim) / dim ** 0.5, rnd(n, kv_heads, dim) / dim ** 0.5, rnd(n, heads, vdim)
    if "delta" in rule:
        k = torch.nn.functional.normalize(k, dim=-1)
    rate = lambda *s: keep + (1 - keep) * torch.rand(*s, generator=g)
    decay = rate(heads) if "constant" in rule else rate(n, heads)
    beta = torch.rand(n, heads, generator=g) if "delta" in rule or rule == "selective" else None
    skip = rnd(heads) if rule == "selective" else None
    return q, k, v, decay, beta, skip


def run(rule, lay, kv_heads, data, rows, lens, slots, chunks):
    from yalis_b200.ops.recurrent import state_scan
    q, k, v, decay, beta, skip = (None if t is None else t.to(DEV) for t in data)
    starts = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    return state_scan(q.flatten(1), k.flatten(1), v.flatten(1), rows, lay, starts, torch.tensor(slots, dtype=torch.int32, device=DEV),
                      kv_heads=kv_heads, decay=decay, beta=beta, max_q_len=max(lens), selective=rule == "selective", skip=skip,
                      chunks=chunks).view(-1, lay.heads, lay.vdim)


def exact(rule, data, first, a, b, heads, kv_heads):
    q, k, v, decay, beta, skip = (None if t is None else t.double() for t in data)
    cut = lambda t: None if t is None else t[a:b]
    d = decay.view(1, heads, 1).expand(b - a, heads, 1) if decay.dim() == 1 else decay[a:b, :, None]
    wide = lambda t: t[a:b].repeat_interleave(heads // kv_heads, 1)
    return walk(first, wide(q), wide(k), cut(v), d, cut(beta), None, None, rule == "selective", skip)


@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("heads,kv_heads,vdim,keep", [(3, 3, 128, 0.5), (4, 2, 20, 0.9), (2, 1, 64, 0.999), (6, 1, 4, 0.0)])
def test_against_a_walk(rule, heads, kv_heads, vdim, keep):
    from yalis_b200.ops.recurrent import StateLayout
    g = torch.Generator().manual_seed(heads * vdim)
    from yalis_b200.ops.recurrent import CHUNKS_FROM
    f = CHUNKS_FROM[{"selective": 3}.get(rule, int("delta" in rule))]
    lens, slots = [1, f, f + 1, f - 1, 0, f + 72, f + 15, 17], [3, 0, 7, 1, 5, 2, 4, 6]
    lay = StateLayout(heads, 128, vdim, conv_channels=3, taps=3)
    data = inputs(rule, heads, kv_heads, vdim, lens, g, keep)
    rows = torch.randn(9, lay.total, generator=g)
    got_rows, plain_rows = rows.to(DEV), rows.to(DEV)
    got = run(rule, lay, kv_heads, data, got_rows, lens, slots, True)
    plain = run(rule, lay, kv_heads, data, plain_rows, lens, slots, False)
    state = lambda r, i: r[slots[i], :lay.state_floats].cpu().view(heads, vdim, 128).double().transpose(1, 2)
    a = 0
    for i, l in enumerate(lens):
        b = a + l
        if l < f:                                  # left to the walk token by token
            assert torch.equal(got[a:b], plain[a:b]) and torch.equal(got_rows[slots[i]], plain_rows[slots[i]])
        else:
            want, last = exact(rule, data, state(rows, i), a, b, heads, kv_heads)
            err, err0 = (got[a:b].cpu().double() - want).norm() / want.norm(), (plain[a:b].cpu().double() - want).norm() / want.norm()
            # 32-bit sums of 128 terms carried over up to 600 tokens
            assert err < 1e-6, (i, err, err0)
            assert (state(got_rows, i) - last).norm() < 1e-6 * last.norm(), i
            alone_rows = rows.to(DEV)
            alone = run(rule, lay, kv_heads, [None if t is None else t if t.dim() == 1 else t[a:b] for t in data], alone_rows, [l], [slots[i]], True)
            assert torch.equal(alone, got[a:b]) and torch.equal(alone_rows[slots[i]], got_rows[slots[i]])
        a = b
    assert torch.equal(got_rows[8], rows[8].to(DEV))
    tail = got_rows[:, lay.state_floats:].cpu()
    assert torch.equal(tail, rows[:, lay.state_floats:])


@pytest.mark.parametrize("rule", RULES)
def test_a_long_portion_is_no_further_off_than_the_walk(rule):
    """2,048 tokens with slow decays: what a rounded decay per chunk would add up to."""
    from yalis_b200.ops.recurrent import StateLayout
    g = torch.Generator().manual_seed(5)
    heads, vdim, n = 4, 32, 2048
    lay = StateLayout(heads, 128, vdim)
    data = inputs(rule, heads, heads, vdim, [n], g, 0.995)
    if "constant" in rule:
        data = data[:3] + (torch.tensor([0.9993, 0.99, 0.9999, 1.0]),) + data[4:]
    want, last = exact(rule, data, torch.zeros(heads, 128, vdim, dtype=torch.float64), 0, n, heads, heads)
    errors = []
    for chunks in (True, False):
        rows = torch.zeros(1, lay.total, device=DEV)
        got = run(rule, lay, heads, data, rows, [n], [0], chunks).cpu().double()
        kept = rows[0, :lay.state_floats].cpu().view(heads, vdim, 128).double().transpose(1, 2)
        errors.append((float((got - want).norm() / want.norm()), float((kept - last).norm() / last.norm())))
    print(rule, errors)
    assert errors[0][0] < max(1.1 * errors[1][0], 3e-7) and errors[0][1] < max(1.1 * errors[1][1], 3e-7), errors


def test_what_is_not_finite_reaches_later_tokens_only():
    from yalis_b200.ops.recurrent import StateLayout
    g = torch.Generator().manual_seed(1)
    lay, n = StateLayout(2, 128, 32), 528
    for rule in RULES:
        data = inputs(rule, 2, 2, 32, [n], g)
        plain = run(rule, lay, 2, data, torch.zeros(1, lay.total, device=DEV), [n], [0], True)
        v = data[2].clone()
        v[70, 1, 5] = float("inf")
        got = run(rule, lay, 2, data[:2] + (v,) + data[3:], torch.zeros(1, lay.total, device=DEV), [n], [0], True)
        assert torch.equal(got[:70], plain[:70]) and torch.equal(got[:, 0], plain[:, 0])
        assert torch.equal(got[:, 1, :5], plain[:, 1, :5]) and not bool(got[70:, 1, 5].isfinite().any())


def test_a_query_that_is_not_finite_reaches_its_own_token_only():
    """The dot products of a chunk's tokens are formed from parts, which an infinity does not have."""
    from yalis_b200.ops.recurrent import StateLayout
    g = torch.Generator().manual_seed(2)
    lay, n = StateLayout(2, 128, 32), 203
    for rule in RULES:
        data = inputs(rule, 2, 2, 32, [n], g)
        plain = run(rule, lay, 2, data, torch.zeros(1, lay.total, device=DEV), [n], [0], True)
        q = data[0].clone()
        q[70, 1, 5] = float("inf")
        got = run(rule, lay, 2, (q,) + data[1:], torch.zeros(1, lay.total, device=DEV), [n], [0], True)
        assert torch.equal(got[:70], plain[:70]) and torch.equal(got[71:], plain[71:]) and torch.equal(got[:, 0], plain[:, 0])
        assert not bool(got[70, 1].isfinite().any())


@pytest.mark.parametrize("rule,lens,bound", [("constant", [150], 256), ("delta", [100], 128), ("selective", [150], 256), ("token", [191, 1, 192], 256),
                                             ("delta", [127, 128, 33], 256), ("selective", [207, 208], 256), ("delta constant", [300], 128)])
def test_a_bound_above_or_below_the_portions_leaves_nobody_out(rule, lens, bound):
    """What a recording gives instead of the longest portion: what each length gives alone, in the form that its own length chooses (a
    portion that is longer than the bound walks)."""
    from yalis_b200.ops.recurrent import StateLayout, state_scan
    g = torch.Generator().manual_seed(sum(lens))
    heads, kv_heads, vdim = 4, 2, 36
    lay, n, slots = StateLayout(heads, 128, vdim), sum(lens), list(range(len(lens)))[::-1]
    q, k, v, decay, beta, skip = (None if t is None else t.to(DEV) for t in inputs(rule, heads, kv_heads, vdim, lens, g))
    first = torch.randn(len(lens), lay.total, generator=g).to(DEV)
    starts = torch.tensor([0] + lens).cumsum(0)

    def run_with(a, b, lens, slots, rows, **how):
        cut = lambda t: None if t is None else t if t.dim() == 1 else t[a:b]
        return state_scan(cut(q).flatten(1), cut(k).flatten(1), cut(v).flatten(1), rows, lay, torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV),
                          torch.tensor(slots, dtype=torch.int32, device=DEV), kv_heads=kv_heads, decay=cut(decay), beta=cut(beta),
                          selective=rule == "selective", skip=skip, **how)

    rows = first.clone()
    got = run_with(0, n, lens, slots, rows, max_q_len=bound, chunks=True)
    want_rows = first.clone()
    for l, a, slot in zip(lens, starts.tolist(), slots):
        want = run_with(a, a + l, [l], [slot], want_rows, max_q_len=l, chunks=l <= bound)
        assert torch.equal(got[a:a + l], want)
    assert torch.equal(rows, want_rows) and not bool((rows == first).all(1).any())


MODELS = [
          ("tirezen_models", {"architecture": "Tirezen", "width": 256, "vocab": 320, "norm": {"eps": 1e-5}, "layers": [
              {"type": "delta", "mixer": {"heads": 2, "kv_heads": 1, "dim": 128, "vdim": 128, "conv": 4}, "mlp": {"kind": "dense", "ff": 256}},
              {"type": "retention", "mixer": {"heads": 2, "dim": 128, "vdim": 128, "decay": [0.96, 0.99], "rot": {"dims": 128, "base": 10000.0}},
               "mlp": {"kind": "dense", "ff": 256}}]}, lengths) for lengths in ([100, 128, 127, 65], [150, 192, 191, 140])] + [
          ("ludelorn_models", {"architecture": "Ludelorn", "embedding": {"scale": 8.0}, "norm": {"eps": 1e-6}, "width": 256, "vocab": 320, "layers": [
              {"type": "parallel", "mixer": {
                  "left": {"heads": 2, "kv_heads": 1, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 64},
                           "rot": {"dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}},
                  "right": {"heads": 4, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}}, "mlp": {"kind": "dense", "ff": 256}}]},
           [200, 208, 207, 193])]


@pytest.mark.parametrize("order", [1, -1])
@pytest.mark.parametrize("module,config,lengths", MODELS, ids=lambda x: x if isinstance(x, str) else "")
def test_a_prompt_from_a_recording_is_the_launched_one(module, config, lengths, order, tmp_path):
    """One request a step, its portion shorter than the recording's bound, at and around the length from which chunks are taken; ten more
    tokens read the state that the prompt left.  All lengths share one recording."""
    import importlib

    from yalis_b200.engine.engine import Engine, StepEntry
    folder = importlib.import_module(module).write_model(config, str(tmp_path), 3)
    eng = Engine(folder, dtype="bfloat16", page_size=16, cache_tokens=1024, max_slots=2)
    g = torch.Generator().manual_seed(4)
    prompt, more = (torch.randint(0, 320, (m,), generator=g).tolist() for m in (max(lengths), 10))

    def logits(length, graphs):
        eng.add_request("r")
        out = eng.run([StepEntry("r", prompt[:length], [length * i // 8 - 1 for i in range(1, 9)])], graphs=graphs)
        rows, replayed = [out.logits.clone()], out.captured
        rows += [eng.run([StepEntry("r", [t], [0])], graphs=False).logits.clone() for t in more]
        eng.finish_request("r")
        return torch.cat(rows), replayed

    for length in lengths[::order]:
        want = logits(length, False)[0]
        replays = 0
        for _ in range(3):
            got, replayed = logits(length, True)
            replays += replayed
            # the recording's padded rows may take the library's products to another kernel: bfloat16 roundings
            assert float((got - want).norm() / want.norm()) < 1e-2, length
        assert replays >= 2


@pytest.mark.parametrize("keep", [0.0, 0.5, 0.9, 0.995])
@pytest.mark.parametrize("rule", RULES)
def test_errors_are_no_larger_than_the_walks(rule, keep):
    """Decays from ``keep`` up to 1, fast ones above all: there the walk rounds little and what the tensor cores cut off shows."""
    from yalis_b200.ops.recurrent import StateLayout
    heads, vdim, n = 16, 64, 256
    lay, squares = StateLayout(heads, 128, vdim), torch.zeros(2, 2, dtype=torch.float64)
    for seed in range(4):
        g = torch.Generator().manual_seed(seed)
        data = inputs(rule, heads, heads, vdim, [n], g, keep)
        on = [None if t is None else t.to(DEV) for t in data]
        want, last = exact(rule, on, torch.zeros(heads, 128, vdim, dtype=torch.float64, device=DEV), 0, n, heads, heads)
        for i, chunks in enumerate((True, False)):
            rows = torch.zeros(1, lay.total, device=DEV)
            got = run(rule, lay, heads, data, rows, [n], [0], chunks).double()
            kept = rows[0, :lay.state_floats].view(heads, vdim, 128).double().transpose(1, 2)
            squares[i] += torch.stack([((got - want).norm() / want.norm()) ** 2, ((kept - last).norm() / last.norm()) ** 2]).cpu()
    errors = squares.sqrt()
    # (five per cent: the spread of such sums over the seeds)
    assert bool((errors[0] <= 1.05 * errors[1]).all()), errors / 2


@pytest.mark.parametrize("what", ["state", "key", "largest", "tiny", "least"])
@pytest.mark.parametrize("rule", RULES)
def test_values_that_parts_cannot_hold(rule, what):
    """Infinities, values that round to one and very small ones: what the walk gives, and the columns beside them as they were."""
    from yalis_b200.ops.recurrent import StateLayout
    g = torch.Generator().manual_seed(7)
    heads, vdim, n = 2, 32, 300
    lay = StateLayout(heads, 128, vdim)
    q, k, v, decay, beta, skip = inputs(rule, heads, heads, vdim, [n], g, 0.8)
    first = torch.randn(1, lay.total, generator=g)
    plain_rows = first.to(DEV)
    plain = run(rule, lay, heads, (q, k, v, decay, beta, skip), plain_rows, [n], [0], True)
    k, v, untouched = k.clone(), v.clone(), torch.ones(heads, vdim, dtype=torch.bool)
    state = first[0, :lay.state_floats].view(heads, vdim, 128)
    if what == "state":
        state[1, 5, 77], untouched[1, 5] = float("inf"), False
    elif what == "key":
        k[250, 1, 9], untouched[1] = float("inf"), False
    elif what == "largest":
        v[100, 1, 5], untouched[1, 5] = 3.4e38, False
    else:                                          # a whole head: about 2^-120, or below the normal numbers
        size = 1e-36 if what == "tiny" else 1e-41
        v[:, 1] *= size
        state[1] *= size
        untouched[1] = False
    data = (q, k, v, decay, beta, skip)
    rows, walk_rows = first.to(DEV), first.to(DEV)
    got, want = run(rule, lay, heads, data, rows, [n], [0], True), run(rule, lay, heads, data, walk_rows, [n], [0], False)
    cut = lambda r: r[0, :lay.state_floats].view(heads, vdim, 128)
    assert torch.equal(got[:, untouched], plain[:, untouched]) and torch.equal(cut(rows)[untouched], cut(plain_rows)[untouched])
    for a, b in ((got, want), (cut(rows), cut(walk_rows))):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a[b.isinf()], b[b.isinf()])
        a, b = (x.double().masked_fill(~b.isfinite(), 0) for x in (a, b))
        if what in ("tiny", "least"):
            # float32 sums in two orders; below the normal numbers a rounding is half of 1.4e-45 at each of some hundred terms
            error = (a - b)[..., 1, :] if a.shape[0] == n else (a - b)[1]
            assert float(error.norm()) <= 1e-6 * float((b[:, 1] if b.shape[0] == n else b[1]).norm()) + 1e-43 * error.numel() ** 0.5
        else:
            assert float((a - b).norm()) <= 1e-5 * float(b.norm())


@pytest.mark.parametrize("rule", ["constant", "delta", "selective"])
@pytest.mark.parametrize("room", [1, 7, 20, 64])
def test_a_step_in_several_launches_has_the_same_bits(rule, room, monkeypatch):
    """Fewer chunks than the step has, or even a portion: what is left goes in further launches, from the state that the last one left."""
    from yalis_b200.ops import recurrent
    g = torch.Generator().manual_seed(room)
    heads, kv_heads, vdim, lens, slots = 4, 2, 36, [300, 3, 0, 256, 513, 209, 1], [2, 0, 3, 6, 1, 5, 4]
    lay = recurrent.StateLayout(heads, 128, vdim)
    data, first = inputs(rule, heads, kv_heads, vdim, lens, g), torch.randn(7, lay.total, generator=g).to(DEV)
    rows, few_rows = first.clone(), first.clone()
    whole = run(rule, lay, kv_heads, data, rows, lens, slots, True)
    monkeypatch.setattr(recurrent, "CHUNK_BYTES", (room - 1) * kv_heads * 2 * 3 * 16 * 128 * 2)
    few = run(rule, lay, kv_heads, data, few_rows, lens, slots, True)
    assert torch.equal(few, whole) and torch.equal(few_rows, rows)


@pytest.mark.parametrize("kind,params", [
    ("retention", {"hidden_size": 64, "heads": 2, "dim": 128, "vdim": 128, "decay": [0.9, 0.99], "rotary": None, "eps": 1e-5}),
    ("gated_delta", {"hidden_size": 64, "heads": 2, "kv_heads": 1, "dim": 128, "vdim": 128, "conv": 4, "eps": 1e-5, "decay": "head"}),
    ("state_space", {"hidden_size": 64, "heads": 4, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1, "eps": 1e-5})])
def test_a_part_can_be_told_to_walk(kind, params):
    """Then a position's result has the same bits however a request is cut; the chunks agree with it to a rounding."""
    from ctx_helper import make_context
    from yalis_b200.config.spec import PartSpec
    from yalis_b200.parts.base import SlotStateCache, make_part
    n, results = 500, {}
    for by_chunks in (False, True):
        part = make_part("mixer", PartSpec(kind, {**params, "by_chunks": by_chunks}))
        g = torch.Generator().manual_seed(2)
        part.load({name: (0.3 * torch.randn(ps.shape, generator=g)).to(DEV, torch.float32 if ps.keep_float32 else torch.bfloat16)
                   for name, ps in part.param_specs().items()})
        z = torch.randn(n, part.in_weight().shape[0], generator=g).to(DEV, torch.bfloat16)
        for cut in ([n], [300, 200], [1, 299, 2, 198]):
            cache = SlotStateCache(torch.zeros(1, part.layout.total, device=DEV))
            y, a = torch.empty(n, part.hidden_width, dtype=torch.bfloat16, device=DEV), 0
            for c in cut:
                ctx, _ = make_context([c], [a], 16)
                part.mix(z[a:a + c], ctx, cache, y[a:a + c])
                a += c
            results.setdefault(by_chunks, []).append((y, cache.state))
    for y, state in results[False]:
        assert torch.equal(y, results[False][0][0]) and torch.equal(state, results[False][0][1])
    assert not torch.equal(results[True][0][1], results[False][0][1])
    for (y, state), (want, last) in zip(results[True], results[False]):
        assert float((y.double() - want.double()).norm()) < 1e-3 * float(want.double().norm()) and float((state - last).norm()) < 1e-6 * float(last.norm())
