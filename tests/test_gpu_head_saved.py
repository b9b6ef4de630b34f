"""The LM head's gradient of the rows, saved in the forward, where a saved-tensor hook hands it back in fp32."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_saved_gradient_in_another_type():
    from composed_mixture_of_experts_engine_b200.models.decoder import lm_head_loss

    got = []
    for unpack in (lambda t: t, lambda t: t.float() if t.dtype == torch.bfloat16 else t):
        g = torch.Generator(device="cuda").manual_seed(1)
        h, w = (torch.randn(s, device="cuda", generator=g).to(torch.bfloat16).requires_grad_() for s in ((70, 64), (512, 64)))
        targets = torch.randint(0, 512, (70,), device="cuda", generator=g)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            loss = lm_head_loss(h, w, targets, 1 / 70)
        (loss * 3.0).backward()  # 3 is exact in bf16, so either form rounds the same products once
        got.append((h.grad, w.grad))
    for a, b in zip(*got):
        assert a.dtype == torch.bfloat16 and a.any() and torch.equal(a, b)
