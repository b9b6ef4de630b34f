"""The router's backward with saved tensors that a hook hands back as views at odd offsets (an offload into one flat buffer)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_backward_with_saved_tensors_at_odd_offsets():
    from composed_mixture_of_experts_engine_b200.ops.moe_router import MoERouter

    torch.manual_seed(0)
    router = MoERouter(256, 64, 4, dtype=torch.bfloat16).cuda()
    x = torch.randn(300, 256, device="cuda").to(torch.bfloat16)

    def grads(pack, unpack):
        router.gate_w.grad = None
        xi = x.clone().requires_grad_()
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            _, w, _ = router(xi)
            (w.float().square().sum() + router.last_aux_loss + router.last_z_loss).backward()
        return xi.grad, router.gate_w.grad.clone()

    def shifted(t):
        if t.dtype == torch.bfloat16:  # the GEMMs' operands: tensor maps refuse what is not aligned
            return t
        flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)[1:]
        return flat.view(t.shape).copy_(t)

    for a, b in zip(grads(lambda t: t, lambda t: t), grads(lambda t: t, shifted)):
        assert torch.equal(a, b)
