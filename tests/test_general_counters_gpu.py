"""General attention layers count in memory of their own call: nothing that another stream, a larger step or a recording shares."""

import pytest
import torch

from ctx_helper import make_context

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PARAMS = {"hidden_size": 256, "num_heads": 16, "num_kv_heads": 8, "head_dim": 64, "window": 96, "sink": True}


class Layer:
    """One layer, its cache and a step of it."""

    def __init__(self, q_lens, before, seed):
        from yalis_b200.config.spec import PartSpec
        from yalis_b200.parts.base import PagedKVCache, make_part
        g = torch.Generator().manual_seed(seed)
        self.part = make_part("mixer", PartSpec("general_attention", PARAMS))
        self.part.load({n: (torch.randn(ps.shape, generator=g) * 0.1).to(torch.float32 if ps.keep_float32 else torch.bfloat16).to(DEV)
                        for n, ps in self.part.param_specs().items()})
        self.ctx, pages = make_context(q_lens, before, 16, seed=seed)
        pool = lambda: torch.randn(pages, 8, 16, 64, generator=g).to(torch.bfloat16).to(DEV)
        self.cache = PagedKVCache(pool(), pool(), "kv_all")
        self.x = torch.randn(sum(q_lens), 256, generator=g).to(torch.bfloat16).to(DEV)

    def __call__(self):
        return self.part.forward(self.x, self.ctx, self.cache)


STEPS = {"decode": ([1] * 70, [31 * i % 700 for i in range(70)]), "prompt": ([300, 77, 1, 513], [0, 100, 640, 0])}


@pytest.mark.parametrize("step", STEPS)
def test_no_shared_counters(step, monkeypatch):
    from yalis_b200.ops import attention as ops
    layer = Layer(*STEPS[step], seed=1)

    def shared(*args):
        raise AssertionError("counters that calls share")

    monkeypatch.setattr(ops, "_tickets", shared)
    monkeypatch.setattr(ops, "_work_counters", shared)
    before = dict(ops.LAUNCHED)
    layer()
    taken = "decode_lean" if step == "decode" else "prefill_tcgen05"
    assert ops.LAUNCHED[taken] == before.get(taken, 0) + 1


@pytest.mark.parametrize("step", STEPS)
def test_two_streams_at_once(step):
    layers = [Layer(*STEPS[step], seed=s) for s in (2, 3)]
    alone = [layer().clone() for layer in layers]
    streams = [torch.cuda.Stream() for _ in layers]
    torch.cuda.synchronize()
    results = [[], []]
    for _ in range(40):
        for i, layer in enumerate(layers):
            with torch.cuda.stream(streams[i]):
                results[i].append(layer())
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(r, alone[i]) for r in results[i])


def test_a_recording_counts_on_after_a_larger_step():
    """A recorded step of few requests, then one of more (request, KV head) pairs than any buffer made for it, and memory given
    out in between: the replay gives the recorded step's result."""
    small, large = Layer([1] * 3, [600, 50, 333], seed=4), Layer([1] * 600, [7 * i % 90 for i in range(600)], seed=5)
    want = small().clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = small()
    large()
    junk = [torch.full((5000,), 7, dtype=torch.int32, device=DEV) for _ in range(20)]
    for _ in range(3):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    assert all(bool((j == 7).all()) for j in junk)
