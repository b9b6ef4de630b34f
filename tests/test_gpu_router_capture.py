"""Routing statistics of captured graphs: each graph brings its own zeroed workspace, so neither the order of replays nor
what the graph pool's memory held before matters, and eager calls afterwards are not touched by it."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["ab", "ba"])
def test_statistics_of_two_graphs(order):
    from composed_mixture_of_experts_engine_b200.ops.moe_router import fused_router_forward

    torch.manual_seed(5)
    N, H, E, K = 300, 256, 16, 2
    w = torch.randn(H, E, device="cuda").to(torch.bfloat16)
    xs = [torch.randn(N, H, device="cuda").to(torch.bfloat16) for _ in range(2)]
    stream, pool = torch.cuda.Stream(), torch.cuda.graph_pool_handle()

    def stats(out):
        return [t.clone() for t in (out.counts, out.counts64, out.mean_prob, out.stats)]

    want = [stats(fused_router_forward(x, w, K)) for x in xs]  # warm-up on another stream than the capture's
    poison, graphs, outs = torch.cuda.CUDAGraph(), {}, {}
    with torch.cuda.graph(poison, pool=pool, stream=stream):
        junk = [torch.full((1024,), 0x3F3F3F3F, device="cuda", dtype=torch.int32) for _ in range(256)]
        del junk
    for name, x in zip("ab", xs):
        graphs[name] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[name], pool=pool, stream=stream):
            outs[name] = fused_router_forward(x, w, K)
    poison.replay()  # fills the memory that the two graphs share with garbage
    for name in order + order[::-1]:
        graphs[name].replay()
        for a, b in zip(stats(outs[name]), want["ab".index(name)]):
            assert torch.equal(a, b)
    with torch.cuda.stream(stream):  # an eager call on the stream of the captures
        for a, b in zip(stats(fused_router_forward(xs[0], w, K)), want[0]):
            assert torch.equal(a, b)
    torch.cuda.synchronize()
