"""The backward of the weighted combine in one pass against the two kernels that it stands for: the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,H,E,capacity", [
    (1, 1, 8, 1, 0),          # one vector
    (130, 8, 512, 16, 0),     # every lane a whole number of pieces
    (257, 6, 1032, 64, 0),    # a ragged last piece, the next size of the kernel
    (64, 40, 264, 48, 0),     # more picks than a warp has lanes
    (1000, 2, 2048, 8, 40),   # most slots dropped
    (33, 4, 4096, 8, 0),      # the widest row
    (1535, 3, 2048, 8, 0),    # the last count of tokens whose picks two warps share, an odd number of picks
    (1536, 3, 2048, 8, 0),    # the first that one warp takes
])
@pytest.mark.parametrize("need_weight", [True, False])
def test_combine_grad(N, K, H, E, capacity, need_weight):
    from composed_mixture_of_experts_engine_b200.ops import _ext, kernels

    g = torch.Generator(device="cuda").manual_seed(N + K + H)
    idx = torch.rand(N, E, device="cuda", generator=g).topk(K, 1).indices.int().contiguous()
    plan = kernels.moe_plan(idx, E, capacity=capacity)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    dy, rows, w = mk(N, H), mk(plan.cap_rows, H), torch.rand(N, K, device="cuda", generator=g)
    n = int(plan.group_offsets[-1])
    want, got = torch.full((plan.cap_rows, H), 7.0, device="cuda", dtype=torch.bfloat16), None
    got = want.clone()
    kernels.gather_rows(dy, plan, slot_scale=w.reshape(-1), out=want)
    dw = torch.full((N, K), 7.0, device="cuda") if need_weight else None
    _ext.ext().combine_grad(dy, plan.slot_row, K, plan.group_offsets, plan.counts_kept, w, rows, got, dw)
    assert torch.equal(got[:n], want[:n]) and bool((got[n:] == 7).all())
    if need_weight:
        assert torch.equal(dw, kernels.combine_bwd_w(rows, plan, dy))
