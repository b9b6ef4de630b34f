"""Tokens' rows copied to their places in expert order, against index arithmetic: exact, since nothing is computed."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,H,E,capacity,pad_src,pad_out", [
    (1, 1, 8, 1, 0, 0, 0),           # one row of one vector
    (3, 2, 1024, 8, 0, 0, 0),        # one whole piece of columns
    (130, 8, 1032, 16, 0, 0, 8),     # a piece and one vector; padded output rows
    (257, 6, 2040, 64, 0, 24, 0),    # ragged second piece; strided source rows
    (64, 40, 264, 48, 0, 0, 0),      # more picks than a warp has lanes
    (1000, 2, 256, 8, 40, 0, 0),     # most slots dropped
])
@pytest.mark.parametrize("zero_padding", [True, False])
def test_place_rows(N, K, H, E, capacity, pad_src, pad_out, zero_padding):
    from composed_mixture_of_experts_engine_b200.ops import _ext, kernels

    g = torch.Generator(device="cuda").manual_seed(N + K + H)
    idx = torch.rand(N, E, device="cuda", generator=g).topk(K, 1).indices.int().contiguous()
    plan = kernels.moe_plan(idx, E, capacity=capacity)
    src = torch.randn(N, H + pad_src, device="cuda", generator=g).to(torch.bfloat16)[:, :H]
    out = torch.full((plan.cap_rows + 1, H + pad_out), 7.0, device="cuda", dtype=torch.bfloat16)
    _ext.ext().place_rows(src, plan.slot_row, K, plan.group_offsets, plan.counts_kept, out[: plan.cap_rows, :H], zero_padding)
    want = torch.full_like(out, 7.0)
    if zero_padding:
        want[: int(plan.group_offsets[-1]), :H] = 0
    slot_row = plan.slot_row.long()
    kept = (slot_row >= 0).nonzero().flatten()
    assert kept.numel() == int(plan.counts_kept.sum())
    want[slot_row[kept], :H] = src[kept // K]
    assert torch.equal(out, want)
