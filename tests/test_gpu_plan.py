"""The row plan at the edges of its launch shapes (one CTA, several units, scanned histograms, bins beyond shared memory)
against a stable sort on the CPU."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,E,cap,lo,n_local", [
    (1, 1, 8, 0, 0, 8),           # one slot
    (30, 4, 700, 0, 0, 700),      # one CTA, many experts
    (4096, 2, 64, 0, 0, 64),      # the last size of the one-CTA launch
    (4097, 2, 64, 0, 16, 16),     # two launches, experts of one rank only
    (5000, 8, 64, 100, 0, 64),    # capacity per (expert, k)
    (40000, 8, 256, 0, 0, 256),   # units x bins beyond the redundant sums: scan launch
    (3000, 8, 1024, 5, 0, 1024),  # bins beyond shared memory
])
def test_plan_matches_a_stable_sort(N, K, E, cap, lo, n_local):
    from composed_mixture_of_experts_engine_b200.ops import kernels

    torch.manual_seed(N)
    bias = torch.randn(E, device="cuda") * 0.7  # uneven load
    idx = (torch.randn(N, E, device="cuda") + bias).topk(K, -1).indices.to(torch.int32)
    plan = kernels.moe_plan(idx, E, expert_lo=lo, n_local=n_local, capacity=cap)
    flat = idx.cpu().flatten().long() - lo
    slots = torch.arange(N * K)
    want_row = torch.full((N * K,), -1)
    off, kept, offs, tiles = 0, [], [], []
    order = torch.argsort(flat * (K if cap else 1) + (slots % K if cap else 0), stable=True)
    bounds = torch.searchsorted(flat[order].contiguous(), torch.arange(n_local + 1))
    for e in range(n_local):
        mine = order[bounds[e]:bounds[e + 1]]
        if cap:  # rows ordered by (expert, k, token), at most `cap` of each (expert, k)
            mine = torch.cat([mine[mine % K == k][:cap] for k in range(K)])
        want_row[mine] = off + torch.arange(mine.numel())
        offs.append(off)
        kept.append(mine.numel())
        n = (mine.numel() + 127) // 128
        tiles += [e] * n
        off += n * 128
    assert torch.equal(plan.slot_row.cpu().long(), want_row)
    want_slot = torch.full((plan.cap_rows,), -1)
    want_slot[want_row[want_row >= 0]] = slots[want_row >= 0]
    assert torch.equal(plan.row_slot.cpu().long(), want_slot)
    assert plan.group_offsets.tolist() == offs + [off] and plan.counts_kept.tolist() == kept
    assert int(plan.num_m_tiles) == off // 128
    assert plan.tile_group.tolist() == tiles + [-1] * (plan.cap_rows // 128 - len(tiles))
