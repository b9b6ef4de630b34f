"""The tables of the expert layer's own row plan against a stable sort on the CPU, with and without dropping, and the layer
in inference with several picks per token and dropping against its training forward."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def routing(N, K, E, seed):
    torch.manual_seed(seed)
    bias = torch.randn(E, device="cuda") * 0.7  # uneven load
    return (torch.randn(N, E, device="cuda") + bias).topk(K, -1).indices.to(torch.int32)


@pytest.mark.parametrize("N,K,E,cap", [
    (1, 1, 8, 0), (64, 8, 64, 0), (300, 4, 8, 0), (300, 4, 8, 20), (4096, 2, 16, 300), (3000, 8, 64, 0), (3000, 8, 64, 90),
    (400, 8, 1024, 3),
])
def test_tables_match_a_stable_sort(N, K, E, cap):
    from composed_mixture_of_experts_engine_b200.ops import _ext, debug, kernels

    idx = routing(N, K, E, N + cap)
    overflow = kernels.overflow_counter(idx.device)
    plan = _ext.ext().moe_local_plan(idx, E, cap, overflow)
    t = _ext.ext().moe_local_tables(plan, N * K, E)
    debug.check_plan(**t, n_local=E, cap_rows=t["row_slot"].numel())
    flat = idx.cpu().flatten().long()
    kept, tiles = [], []
    for e in range(E):
        mine = torch.nonzero(flat == e).flatten()
        if cap:
            mine = torch.cat([mine[mine % K == k][:cap] for k in range(K)])
        kept.append(mine.numel())
        tiles.append((mine.numel() + 127) // 128)
        row0 = 128 * sum(tiles[:-1])
        assert t["slot_row"].cpu().long()[mine].tolist() == list(range(row0, row0 + mine.numel()))
    assert t["counts_kept"].tolist() == kept and int(t["num_m_tiles"]) == sum(tiles)
    assert t["tile_rows"].tolist()[:sum(tiles)] == [min(128, kept[e] - 128 * i) for e in range(E) for i in range(tiles[e])]
    first = [sum(tiles[:e]) for e in range(E)]
    pairs = [2 * (first[e] + i) + (i + 1 == tiles[e]) for e in range(E) for i in range(0, tiles[e], 2)]
    assert int(t["num_pairs"]) == len(pairs) and t["pair_tile"].tolist()[:len(pairs)] == pairs
    assert t["group_order"].tolist() == sorted(range(E), key=lambda e: (-tiles[e], e))
    assert int((t["slot_row"] >= 0).sum()) == sum(kept)


@pytest.mark.parametrize("N,K,E,cap,debug_on", [(40, 4, 16, 0, False), (40, 4, 16, 6, False), (64, 8, 64, 5, True),
                                                (500, 4, 8, 150, True)])
def test_inference_with_dropping_matches_the_training_forward(monkeypatch, N, K, E, cap, debug_on):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops.kernels import check_status

    monkeypatch.setenv("CMOE_DEBUG_BOUNDS", "1" if debug_on else "0")
    H, F = 256, 136
    idx = routing(N, K, E, N)
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda") * scale).to(torch.bfloat16)
    x, w13, w2 = mk(N, H), mk(E, 2 * F, H, scale=H ** -0.5), mk(E, H, F, scale=F ** -0.5)
    gate = torch.rand(N, K, device="cuda") + 0.5
    want = OF.local_moe(x.clone().requires_grad_(), gate, idx, w13, w2, capacity=cap).detach()
    keep = ~OF.capacity_drop_mask_reference(idx, E, cap) if cap else None
    ref = OF.experts_reference(x.double(), idx.long(), gate.double(), w13.double(), w2.double(), 0, keep)
    assert float((want.double() - ref).norm() / ref.norm()) < 1e-2  # three roundings to bf16 (2^-9) in a row
    for _ in range(2):
        junk = [torch.full((n,), float("nan"), device="cuda") for n in (1 << 22, 1 << 20, 1 << 18, 1 << 16)]
        del junk
        with torch.no_grad():
            assert torch.equal(OF.local_moe(x, gate, idx, w13, w2, capacity=cap), want)
    check_status(x.device)
