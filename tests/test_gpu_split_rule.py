"""Where a call's rows are split over several CTAs by itself, that is not the slower way: timed against whole rows in graphs of calls
on either side of the rule's lines, and where a line used to lie too low."""
import numpy as np
import pytest

from mako_b200.sampler import BatchSampler, SamplingParams, pack_params

pytestmark = pytest.mark.gpu

TOP_K = SamplingParams(temperature=0.7, top_k=40, top_p=0.95)
MIN_P = SamplingParams(temperature=0.8, top_p=0.9, min_p=0.05)
GREEDY = SamplingParams(temperature=0.0)


@pytest.mark.parametrize("params,tiles,rows", [
    (GREEDY, 12, 16), (GREEDY, 20, 148), (GREEDY, 37, 148), (TOP_K, 4, 1), (TOP_K, 8, 16), (MIN_P, 12, 96), (MIN_P, 28, 148),
    (MIN_P, 37, 1), ("own", 37, 148), ("own", 20, 4), ("pq", 20, 148), ("pq", 37, 4),
], ids=lambda x: x if isinstance(x, str) else str(x) if isinstance(x, int) else f"t{x.temperature}k{x.top_k}m{x.min_p}")
def test_the_rule_does_not_choose_the_slower_way(params, tiles, rows):
    import torch
    v = tiles * 4096 - 96
    if isinstance(params, str) and params == "own":
        params = torch.from_numpy(pack_params([(TOP_K, MIN_P, GREEDY)[b % 3] for b in range(rows)])).cuda()
    g = torch.Generator(device="cuda")
    g.manual_seed(tiles * 1000 + rows)
    n = max(3, min(32, 60_000_000 // (rows * v)))
    logits = torch.randn((n, rows, v), device="cuda", generator=g) * 2
    at = torch.randint(0, v, (n, rows, 8), device="cuda", generator=g)
    logits.scatter_(2, at, torch.rand((n, rows, 8), device="cuda", generator=g) * 7 + 8)
    u = torch.rand(rows, device="cuda", generator=g)
    s, graphs, times = BatchSampler(v, rows), [], ([], [])

    def call(k):
        if isinstance(params, str):
            return s.verify_pq(logits[k % n], logits[(k + 1) % n], TOP_K, u, u, u)
        return s.sample(logits[k % n], params, u)

    side = torch.cuda.Stream()
    for on in (True, False):
        s.set_split(on)
        with torch.cuda.stream(side):
            call(0)
            side.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                for k in range(4 * n):
                    call(k)
        graphs.append(graph)
    for _ in range(12):
        for graph, t in zip(graphs, times):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
    by_itself, whole = (float(np.median(t[2:])) for t in times)
    assert by_itself < 1.08 * whole, (by_itself / (4 * n) * 1e3, whole / (4 * n) * 1e3)
