"""A router class of a user's own sees what the fused path leaves on the module."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("train", [False, True])
def test_attributes_of_a_subclass_are_set_through_it(train):
    from composed_mixture_of_experts_engine_b200.ops.moe_router import MoERouter

    class Watched(MoERouter):
        @property
        def last_aux_loss(self):
            return self._seen[-1]

        @last_aux_loss.setter
        def last_aux_loss(self, value):
            self.__dict__.setdefault("_seen", []).append(value)

    router = Watched(64, 8, 2, dtype=torch.bfloat16).cuda()
    x = torch.randn(40, 64, device="cuda").to(torch.bfloat16)
    with torch.set_grad_enabled(train):
        router(x)
    assert router.last_profile.used_fused_kernel
    assert len(router._seen) == 2 and router.last_aux_loss is router._seen[-1] and float(router.last_aux_loss.detach()) > 0
