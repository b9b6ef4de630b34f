"""With the bounds checks on, the expert layer's own plan is validated before a kernel reads it: every table, on the path that
runs.  Plain tensors and a stand-in for the native layer, so this runs on the CPU."""

import pytest
import torch

from composed_mixture_of_experts_engine_b200.ops import debug, kernels
from composed_mixture_of_experts_engine_b200.ops import functional as OF


def tables(rows):
    """The plan of one slot per row, experts in order, made with plain tensor ops."""
    E, n = len(rows), sum(rows)
    tiles = [(r + 127) // 128 for r in rows]
    offs = torch.zeros(E + 1, dtype=torch.int64)
    offs[1:] = torch.tensor(tiles).cumsum(0) * 128
    cap = int(offs[-1]) + 128
    row_slot = torch.full((cap,), -1)
    slot_row = torch.cat([int(offs[e]) + torch.arange(r) for e, r in enumerate(rows)])
    row_slot[slot_row] = torch.arange(n)
    group = torch.repeat_interleave(torch.arange(E), torch.tensor(tiles))
    pairs, tile_rows = [], []
    for e, r in enumerate(rows):
        for i in range(tiles[e]):
            tile_rows.append(min(128, r - 128 * i))
            if i % 2 == 0:
                pairs.append(2 * (int(offs[e]) // 128 + i) + (i + 1 == tiles[e]))
    pad = lambda v, m: torch.cat([torch.as_tensor(v), torch.full((m - len(v),), -1)])
    t = dict(slot_row=slot_row, row_slot=row_slot, tile_group=pad(group, cap // 128),
             num_m_tiles=torch.tensor([sum(tiles)]), group_offsets=offs, pair_tile=pad(pairs, cap // 128),
             num_pairs=torch.tensor([len(pairs)]), tile_rows=pad(tile_rows, cap // 128),
             group_order=torch.tensor(sorted(range(E), key=lambda e: (-tiles[e], e))),
             counts_kept=torch.tensor(rows))
    return {k: v.to(torch.int32) for k, v in t.items()}


ROWS = [5, 0, 300, 128, 129]


def test_each_broken_table_is_named():
    good = tables(ROWS)
    args = dict(n_local=len(ROWS), cap_rows=good["row_slot"].numel())
    debug.check_plan(**good, **args)
    for name, pos, value, message in (
            ("pair_tile", 1, 99, r"pair_tile\[1\] = 99"), ("pair_tile", 0, 0, r"pair_tile\[0\] = 0"),
            ("num_pairs", 0, 7, "num_pairs = 7"), ("tile_rows", 0, 4, r"tile_rows\[0\] = 4"),
            ("tile_rows", 3, 129, r"tile_rows\[3\] = 129"), ("group_order", 0, 5, r"group_order\[0\] = 5"),
            ("group_order", 1, 2, "group_order names expert"), ("counts_kept", 2, 299, r"counts_kept\[2\] = 299")):
        bad = {k: v.clone() for k, v in good.items()}
        bad[name][pos] = value
        with pytest.raises(debug.PlanBoundsError, match=message):
            debug.check_plan(**bad, **args)


@pytest.mark.parametrize("broken", ["", "pair_tile", "tile_rows", "group_order", "slot_row"])
def test_the_layer_checks_the_plan_it_uses(monkeypatch, broken):
    class Ext:
        ran = False

        def moe_local_plan(self, idx, E, capacity, overflow):
            return "plan"

        def moe_local_tables(self, plan, n_slots, E):
            t = tables(ROWS)
            if broken:
                t[broken][0] = 1 << 20
            return t

        def moe_local_forward(self, *args):
            assert args[-1] == "plan"
            Ext.ran = True
            return (args[0],) + ("plan",) + (None,) * 4

    monkeypatch.setenv("CMOE_DEBUG_BOUNDS", "1")
    monkeypatch.setattr(OF, "on_device_path", lambda *t: True)
    monkeypatch.setattr(OF._ext, "ext", lambda: Ext())
    monkeypatch.setattr(kernels, "status_word", lambda device: None)
    monkeypatch.setattr(kernels, "overflow_counter", lambda device: None)
    N, E, H, F = sum(ROWS), len(ROWS), 8, 4
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(ROWS))[:, None]
    mk = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    call = lambda: OF.local_moe(mk(N, H), torch.ones(N, 1), idx, mk(E, 2 * F, H), mk(E, H, F))
    if broken:
        with pytest.raises(debug.PlanBoundsError):
            call()
        assert not Ext.ran
    else:
        call()
        assert Ext.ran
