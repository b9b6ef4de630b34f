"""Kernels that may start before their predecessor has ended take plain pointers (csrc/launch.h): a `__restrict__` one may
be read through the non-coherent path or ahead of the wait."""

import re

import pytest

from composed_mixture_of_experts_engine_b200.ops._ext import CSRC_DIR


@pytest.mark.parametrize("name", ["ops.cu", "plan.cu", "router.cu", "gemm.cu", "gemm2.cu"])
def test_chained_kernels_take_plain_pointers(name):
    text = (CSRC_DIR / name).read_text()
    kernels = re.split(r"(?=__global__ void)", text)[1:]
    chained = [k for k in kernels if "chain_wait(" in k]
    assert chained
    for k in chained:
        signature = k[: k.index("{")]
        assert "__restrict__" not in signature, signature


def test_launches_that_wait_for_other_ranks_hold_their_successor_back():
    """A successor that starts early would occupy the SMs while this kernel waits for its peers; `chained` is set by
    `gemm_overlaps_neighbours` (csrc/gemm.cuh), which no launch with a row pull, a scatter or ready flags passes."""
    text = (CSRC_DIR / "gemm.cu").read_text()
    triggers = re.findall(r".*chain_trigger\(\);", text)
    assert triggers and all("if (p.chained)" in line for line in triggers)
    rule = re.search(r"inline bool gemm_overlaps_neighbours\(.*?\{(.*?)\}", (CSRC_DIR / "gemm.cuh").read_text(), re.S).group(1)
    assert all(f"a.{name} == nullptr" in rule for name in ("pull_row_slot", "scatter_row_slot", "ready_flags"))


@pytest.mark.parametrize("name", ["gemm.cu", "gemm2.cu"])
def test_tables_read_ahead_of_the_wait_bypass_l1(name):
    """The warp that loads weights without waiting for the predecessor reads the row plan past L1."""
    text = (CSRC_DIR / name).read_text()
    for table in ("tile_group", "num_m_tiles") if name == "gemm.cu" else ("tile_group", "pair_tile", "num_pairs"):
        assert re.search(rf"ahead \? load_ahead_of_wait\(p\.{table}", text), table
    assert len(re.findall(r"= decode(?:_tile|2)\(.*, ahead\);", text)) == 1
