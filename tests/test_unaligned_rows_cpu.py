"""Token matrices whose rows lie off 16-byte boundaries reach the native expert layer as aligned copies (its row kernels read
16-byte vectors), all others as they are.  The native call is a stand-in, so this runs on the CPU."""

import pytest
import torch

from composed_mixture_of_experts_engine_b200.ops import functional as OF
from composed_mixture_of_experts_engine_b200.ops import kernels

N, H, E, F = 6, 16, 4, 8


def views():
    big = torch.randn(N * H + 8).to(torch.bfloat16)
    wide = torch.randn(N, 2 * H + 4).to(torch.bfloat16)
    return {
        "contiguous": (big[:N * H].view(N, H), False),
        "row stride": (torch.randn(N, 2 * H).to(torch.bfloat16)[:, :H], False),
        "off by one": (big[1:1 + N * H].view(N, H), True),
        "odd row stride": (wide[:, :H], True),
        "column offset": (wide[:, 4:4 + H], True),
    }


@pytest.mark.parametrize("name", list(views()))
def test_layer_input_and_gradient(monkeypatch, name):
    seen = {}

    class Ext:
        def moe_local_forward(self, x, *args):
            seen["x"] = x
            return (x * 2,) + (torch.zeros(8),) * 5

        def moe_local_backward(self, dy, *args):
            seen["dy"] = dy
            return dy * 2, None, None, None

    monkeypatch.delenv("CMOE_DEBUG_BOUNDS", raising=False)
    monkeypatch.setattr(OF, "on_device_path", lambda *t: True)
    monkeypatch.setattr(OF._ext, "ext", lambda: Ext())
    monkeypatch.setattr(kernels, "status_word", lambda device: None)
    monkeypatch.setattr(kernels, "overflow_counter", lambda device: None)
    x, copied = views()[name]
    w13, w2 = torch.zeros(E, 2 * F, H, dtype=torch.bfloat16), torch.zeros(E, H, F, dtype=torch.bfloat16)
    xin = x.detach().requires_grad_()
    y = OF.local_moe(xin, torch.ones(N, 1), torch.zeros(N, 1, dtype=torch.int64), w13, w2)
    got = seen["x"]
    assert got.data_ptr() % 16 == 0 and got.stride(0) % 8 == 0 and got.stride(1) == 1 and torch.equal(got, x)
    assert (got.data_ptr() != xin.data_ptr()) == copied
    dy, _ = views()[name]
    y.backward(dy)
    assert seen["dy"].is_contiguous() and seen["dy"].data_ptr() % 16 == 0 and torch.equal(seen["dy"], dy)
    assert torch.equal(xin.grad, dy * 2)
