"""Kernels whose start overlaps their predecessor: a chain without host waits gives the bits of one that waits after every
call, with inputs that a kernel just before the layer writes and weights that change between the calls."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,H,F,E,K", [(1, 256, 256, 8, 2), (64, 512, 256, 64, 8), (700, 1024, 512, 16, 2)])
def test_layer_calls_in_a_row(tokens, H, F, E, K):
    from composed_mixture_of_experts_engine_b200.parallel import DistributedMoELayer

    def calls(wait):
        torch.manual_seed(3)
        with torch.device("cuda"):
            layer = DistributedMoELayer(H, F, E, K, dtype=torch.bfloat16)
        x = torch.randn(tokens, H, device="cuda").to(torch.bfloat16)
        out = []
        for i in range(12):
            x.mul_(-0.75).add_(0.5)
            xi = x.clone().requires_grad_(i % 2 == 0)
            with torch.set_grad_enabled(i % 2 == 0):
                y = layer(xi)
            if i % 2 == 0:
                y.sum().backward()
                out.append(xi.grad)
            with torch.no_grad():
                for p in layer.parameters():
                    p.mul_(1.0625)
            out.append(y.detach())
            if wait:
                torch.cuda.synchronize()
        return out

    waited, chained = calls(True), calls(False)
    for a, b in zip(waited, chained):
        assert torch.equal(a, b)
