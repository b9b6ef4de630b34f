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
