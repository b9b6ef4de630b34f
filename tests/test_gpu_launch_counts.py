"""The reported number of launched kernels is counted where they are launched, not estimated per call."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_counts_follow_the_launches():
    from composed_mixture_of_experts_engine_b200.ops import _ext, kernels

    def launched(fn):
        fn()
        _ext.reset_launch_counts()
        fn()
        return _ext.launch_counts_total()

    def plan(N, K, E):
        idx = torch.randint(0, E, (N, K), device="cuda", dtype=torch.int32)
        return lambda: kernels.moe_plan(idx, E)

    assert launched(plan(64, 8, 64)) == 1       # one CTA
    assert launched(plan(16384, 8, 64)) == 2    # count, rank
    assert launched(plan(40000, 8, 256)) == 3   # count, scan, rank
    x, w = (torch.randn(64, 64, device="cuda").to(torch.bfloat16) for _ in range(2))
    assert launched(lambda: kernels.linear_nt(x, w)) == 1
    a, b = (torch.randn(8192, 64, device="cuda").to(torch.bfloat16) for _ in range(2))
    assert launched(lambda: kernels.linear_tn(a, b, splits=1)) == 1
    assert launched(lambda: kernels.linear_tn(a, b, splits=4)) == 2  # the pieces and their sum
    assert launched(lambda: None) == 0
