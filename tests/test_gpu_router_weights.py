"""The gate weights and the log-sum-exp are, to the last bit, those of their definition summed in a fixed order (experts
ascending, picks descending), whatever tile, cluster or lane computed them."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,E,K", [
    (1, 64, 8, 1),         # a row of one lane group, top-1
    (300, 256, 64, 8),     # short tiles
    (129, 520, 256, 8),    # experts split over a cluster of four CTAs
    (300, 512, 128, 6),    # clusters of two CTAs
    (1000, 256, 72, 3),    # the smallest expert counts of the two widest lane variants,
    (129, 256, 136, 8),    # whose lanes look past the last expert
    (300, 256, 224, 4),
    (20000, 256, 32, 2),   # full tiles
])
def test_weights_follow_the_definition_to_the_bit(N, H, E, K):
    from composed_mixture_of_experts_engine_b200.ops.moe_router import fused_router_forward, moe_topk_route

    torch.manual_seed(N + E)
    x = torch.randn(N, H, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(H, E, device="cuda") * 2 / H ** 0.5).to(torch.bfloat16)
    out = fused_router_forward(x, w, K)
    lg = out.logits
    mx = lg.max(-1, keepdim=True).values
    ex = torch.exp(lg - mx)
    se = torch.zeros(N, device="cuda")
    for e in range(E):
        se = se + ex[:, e]
    lse = mx[:, 0] + torch.log(se)
    assert torch.equal(out.lse, lse)
    pk = torch.exp(lg.gather(1, out.idx32.long()) - lse[:, None])
    psum = torch.zeros(N, device="cuda")
    for k in range(K):
        psum = psum + pk[:, k]
    want = pk * torch.reciprocal(psum)[:, None]
    assert torch.equal(out.w32, want) and torch.equal(out.w16, want.to(torch.bfloat16))
    assert torch.equal(moe_topk_route(x, w, K)[1], out.w16)
