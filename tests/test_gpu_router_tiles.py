"""The fused router at the edges of its tiles: rows split over clusters, every experts-per-lane variant, ragged token
counts, ties; against the fp64 oracle."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,E,K", [
    (1, 8, 8, 8),          # one token, one k-block, K = E
    (64, 2048, 64, 8),     # short tiles of 16 rows
    (129, 520, 256, 8),    # a cluster of four CTAs per tile, a ragged last k-block, the widest expert variant
    (300, 4096, 128, 6),   # clusters of two CTAs, 128 experts
    (127, 1024, 24, 3),    # expert count that is no multiple of 16
    (8190, 1024, 40, 1),   # tiles of 64 rows
    (20000, 256, 32, 4),   # more row tiles than SMs
])
def test_route_matches_the_oracle_at_tile_edges(N, H, E, K):
    from composed_mixture_of_experts_engine_b200.ops.moe_router import MoERouter, moe_topk_route

    torch.manual_seed(N + E)
    router = MoERouter(H, E, K, dtype=torch.bfloat16).cuda()
    x = torch.randn(N, H, device="cuda", dtype=torch.bfloat16)
    x[N // 2] = 0  # all logits equal: the lowest K experts, in order
    logits = x.double() @ router.gate_w.double()
    p = torch.softmax(logits, -1)
    idx, w = moe_topk_route(x, router.gate_w.detach(), K)            # decision only
    gidx, gw, cnt = router(x.clone().requires_grad_())               # with statistics and gradients
    assert torch.equal(idx, gidx) and torch.equal(w, gw.detach())
    assert idx.dtype == torch.int64 and w.dtype == torch.bfloat16 and cnt.dtype == torch.int64
    assert idx[N // 2].tolist() == list(range(K))
    # picks: distinct, in range, and no probability further from the oracle's than fp32 logits allow (H products of
    # unit variance: error of a logit below 1e-4)
    assert int(idx.min()) >= 0 and int(idx.max()) < E
    assert all(len(set(r)) == K for r in idx[:: max(1, N // 64)].tolist())
    want = torch.topk(p, K, -1).values
    got = p.gather(1, idx)
    assert torch.allclose(got, want, rtol=1e-3, atol=1e-9)
    # weights: one rounding to bf16 (2^-9 relative) on top of the same logit error
    assert torch.allclose(w.double(), got / got.sum(-1, keepdim=True), rtol=2 ** -8, atol=1e-6)
    assert torch.equal(cnt, torch.bincount(idx.flatten(), minlength=E))
    f = cnt.double() / (N * K)
    assert abs(float(router.last_aux_loss) - E * float((f * p.mean(0)).sum())) < 1e-3
    z = float((torch.logsumexp(logits, -1) ** 2).mean())
    assert abs(float(router.last_z_loss) - z) < 1e-3 * max(1.0, z)
    assert router.last_profile.dispatch_counts == cnt.tolist()
