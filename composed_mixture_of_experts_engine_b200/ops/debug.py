"""Debug-time index and memory checks (``CMOE_DEBUG_BOUNDS=1``).

The reference has no sanitizer mode of any kind; its safety nets are run-time asserts on routing results
(pkg/kernels/moe_router.py:693-700, pkg/distributed/moe_layer.py:355-358).  The kernels here take row indices that
other kernels computed (the row plan) and write into memory that other GPUs map, so a debug mode checks both before
anything can go wrong on the device:

* ``check_plan``: every index of a row plan is validated with ordinary tensor ops before a gather / GEMM / combine
  kernel consumes it (slot -> row and row -> slot tables in range and inverse to each other, tile table consistent
  with the expert offsets, live tiles within the buffer).  The first violation raises ``PlanBoundsError`` naming the
  table, the position and the value: the bad index never reaches a kernel.
* ``Canary``: guard bands around a buffer (used for the symmetric buffers that peers write into); ``verify`` reports
  the first guard byte that changed, i.e. a write that left its buffer.

Both cost a host synchronisation per call and are meant for tests and bring-up on small shapes, never for timing.
"""

from __future__ import annotations

import os
from typing import Optional

import torch

GUARD_BYTES = 4096
GUARD_PATTERN = 0xA5


def enabled() -> bool:
    return os.environ.get("CMOE_DEBUG_BOUNDS", "0") not in ("", "0")


class PlanBoundsError(RuntimeError):
    """A row plan holds an index outside its table (the message names table, position and value)."""


class GuardBandError(RuntimeError):
    """Bytes outside a guarded buffer were overwritten."""


def _first_bad(mask: torch.Tensor) -> Optional[int]:
    bad = torch.nonzero(mask.reshape(-1), as_tuple=False)
    return int(bad[0]) if bad.numel() else None


def check_plan(slot_row: torch.Tensor, row_slot: torch.Tensor, tile_group: torch.Tensor, num_m_tiles: torch.Tensor,
               group_offsets: torch.Tensor, n_local: int, cap_rows: int, n_slots: Optional[int] = None,
               pair_tile: Optional[torch.Tensor] = None, num_pairs: Optional[torch.Tensor] = None,
               tile_rows: Optional[torch.Tensor] = None, group_order: Optional[torch.Tensor] = None,
               counts_kept: Optional[torch.Tensor] = None) -> None:
    """Validate one row plan.  ``slot_row`` [n_slots] (row of each (token, k) slot or -1), ``row_slot`` [cap_rows]
    (slot of each row or -1), ``tile_group`` [cap_rows / 128] (expert of each 128-row tile or -1), ``num_m_tiles``
    [1], ``group_offsets`` [n_local + 1].  The tables of the expert layer's own plan, where given: ``pair_tile``
    [cap_rows / 128] / ``num_pairs`` [1] (2 * first tile + 1 if the pair has only that one), ``tile_rows``
    [cap_rows / 128] (live rows of each tile), ``group_order`` [n_local] (experts from most to fewest padded rows),
    ``counts_kept`` [n_local] (live rows of each expert)."""
    n_slots = int(slot_row.numel()) if n_slots is None else n_slots
    tiles = int(num_m_tiles.reshape(-1)[0])
    if tiles < 0 or tiles * 128 > cap_rows or tiles > tile_group.numel():
        raise PlanBoundsError(f"num_m_tiles = {tiles} does not fit a buffer of {cap_rows} rows")
    sr = slot_row.reshape(-1)[:n_slots].long()
    i = _first_bad((sr < -1) | (sr >= tiles * 128))
    if i is not None:
        raise PlanBoundsError(f"slot_row[{i}] = {int(sr[i])} is outside [-1, {tiles * 128})")
    rs = row_slot.reshape(-1)[: tiles * 128].long()
    i = _first_bad((rs < -1) | (rs >= n_slots))
    if i is not None:
        raise PlanBoundsError(f"row_slot[{i}] = {int(rs[i])} is outside [-1, {n_slots})")
    # the two tables are inverse to each other wherever both are set
    live = torch.nonzero(sr >= 0, as_tuple=False).reshape(-1)
    if live.numel():
        back = rs[sr[live]]
        i = _first_bad(back != live)
        if i is not None:
            s = int(live[i])
            raise PlanBoundsError(f"slot {s} maps to row {int(sr[s])}, but that row maps back to slot {int(back[i])}")
    tg = tile_group.reshape(-1)[:tiles].long()
    i = _first_bad((tg < -1) | (tg >= n_local))
    if i is not None:
        raise PlanBoundsError(f"tile_group[{i}] = {int(tg[i])} is outside [-1, {n_local})")
    go = group_offsets.reshape(-1).long()
    if go.numel() != n_local + 1 or int(go[0]) != 0:
        raise PlanBoundsError(f"group_offsets has {go.numel()} entries starting at {int(go[0]) if go.numel() else None}")
    i = _first_bad((go[1:] < go[:-1]) | (go % 128 != 0)[1:] | (go[1:] > cap_rows))
    if i is not None:
        raise PlanBoundsError(f"group_offsets[{i + 1}] = {int(go[i + 1])} (previous {int(go[i])}, buffer {cap_rows})")
    if int(go[-1]) != tiles * 128:
        raise PlanBoundsError(f"group_offsets end at {int(go[-1])} but {tiles} tiles are live")
    # every live tile lies inside the segment of the expert it names
    if tiles:
        t0 = torch.arange(tiles, device=tg.device) * 128
        named = tg.clamp(min=0)
        inside = (t0 >= go[named]) & (t0 < go[named + 1])
        i = _first_bad((tg >= 0) & ~inside)
        if i is not None:
            raise PlanBoundsError(f"tile {i} names expert {int(tg[i])} whose rows are [{int(go[tg[i]])}, "
                                  f"{int(go[tg[i] + 1])})")
    # every expert's live rows lie in front of its padding
    live_rows = (rs >= 0).long()
    before = torch.cat([live_rows.new_zeros(1), live_rows.cumsum(0)])
    per_expert = before[go[1:]] - before[go[:-1]]
    if counts_kept is not None:
        i = _first_bad(counts_kept.reshape(-1).long() != per_expert)
        if i is not None:
            raise PlanBoundsError(f"counts_kept[{i}] = {int(counts_kept.reshape(-1)[i])}, but expert {i} has "
                                  f"{int(per_expert[i])} rows")
    if tile_rows is not None and tiles:
        got = tile_rows.reshape(-1)[:tiles].long()
        per_tile = live_rows.view(tiles, 128)
        want = per_tile.sum(1)
        i = _first_bad(got != want)
        if i is not None:
            raise PlanBoundsError(f"tile_rows[{i}] = {int(got[i])}, but the tile has {int(want[i])} live rows")
        i = _first_bad((per_tile[:, 1:] > per_tile[:, :-1]).any(1))
        if i is not None:
            raise PlanBoundsError(f"tile {i} has a live row behind padding")
    if group_order is not None:
        order, padded = group_order.reshape(-1).long(), go[1:] - go[:-1]
        i = _first_bad((order < 0) | (order >= n_local))
        if i is not None:
            raise PlanBoundsError(f"group_order[{i}] = {int(order[i])} is outside [0, {n_local})")
        i = _first_bad(torch.bincount(order, minlength=n_local) != 1)
        if i is not None:
            raise PlanBoundsError(f"group_order names expert {i} not exactly once")
        i = _first_bad(padded[order][1:] > padded[order][:-1])
        if i is not None:
            raise PlanBoundsError(f"group_order[{i + 1}] = {int(order[i + 1])} has more rows than the expert before it")
    if pair_tile is not None and num_pairs is not None:
        # tiles t of an expert with an even distance from its first one start a pair, alone where no other follows
        t = torch.arange(tiles, device=tg.device)
        first, last = go[tg] // 128, go[tg + 1] // 128 - 1
        starts = (t - first) % 2 == 0
        want = (2 * t + (t == last).long())[starts]
        n = int(num_pairs.reshape(-1)[0])
        if n != want.numel():
            raise PlanBoundsError(f"num_pairs = {n}, but the tiles make {want.numel()} pairs")
        got = pair_tile.reshape(-1)[:n].long()
        i = _first_bad(got != want)
        if i is not None:
            raise PlanBoundsError(f"pair_tile[{i}] = {int(got[i])}, expected {int(want[i])}")


class Canary:
    """Guard bands of ``GUARD_BYTES`` before and after the useful part of a byte buffer."""

    def __init__(self, full: torch.Tensor, nbytes: int):
        if full.dtype != torch.uint8 or full.numel() < nbytes + 2 * GUARD_BYTES:
            raise ValueError("guarded buffers are uint8 tensors with room for both guard bands")
        self.full, self.nbytes = full, nbytes
        self.front = full[:GUARD_BYTES]
        self.back = full[GUARD_BYTES + nbytes: GUARD_BYTES + nbytes + GUARD_BYTES]
        self.front.fill_(GUARD_PATTERN)
        self.back.fill_(GUARD_PATTERN)

    @property
    def inner(self) -> torch.Tensor:
        return self.full[GUARD_BYTES: GUARD_BYTES + self.nbytes]

    def verify(self, name: str = "buffer") -> None:
        for label, band, base in (("before", self.front, -GUARD_BYTES), ("after", self.back, self.nbytes)):
            i = _first_bad(band != GUARD_PATTERN)
            if i is not None:
                raise GuardBandError(f"{name}: byte at offset {base + i} ({label} the buffer) was overwritten "
                                     f"with {int(band[i])}")
