"""The row plan on every device of a process, where its launch needs more shared memory than the default."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices")
def test_plan_on_two_devices():
    from composed_mixture_of_experts_engine_b200.ops import kernels

    torch.manual_seed(1)
    idx = torch.randint(0, 64, (1000, 8), dtype=torch.int32)  # 512 (expert, k) bins: 72 KiB
    plans = []
    for d in (0, 1):
        with torch.cuda.device(d):
            plans.append(kernels.moe_plan(idx.cuda(d), 64, capacity=40))
            torch.cuda.synchronize()
    assert torch.equal(plans[0].slot_row.cpu(), plans[1].slot_row.cpu())
