"""The gate weights inside the expert FFN: the layer's result and the gradient of the weights against float64."""

import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,H,F,E,capacity,slow", [
    (5, 2, 64, 72, 4, 0, False),        # one ragged piece of columns
    (300, 2, 256, 136, 4, 0, False),    # several pieces, the last one ragged
    (700, 4, 128, 264, 8, 0, False),    # a second tile of columns with one group of eight
    (3000, 2, 192, 520, 4, 0, False),   # pairs of tiles, experts with an odd number of them
    (4096, 6, 512, 256, 8, 0, False),
    (2048, 8, 256, 320, 16, 300, False),  # slots dropped: their weights have no gradient
    (900, 2, 128, 200, 4, 0, True),     # stores from registers
])
def test_gate_weight_gradient(N, K, H, F, E, capacity, slow):
    from composed_mixture_of_experts_engine_b200.ops.kernels import check_status

    if slow:  # the switches are read once per process
        code = f"import tests.test_gpu_gate_grad as t; t.check({N}, {K}, {H}, {F}, {E}, {capacity}); print('same')"
        out = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, capture_output=True,
                             env={**os.environ, "CMOE_GEMM_DIRECT_EPILOGUE": "1", "CMOE_GEMM_2CTA": "0"}, text=True, timeout=300)
        assert out.returncode == 0 and "same" in out.stdout, out.stdout + out.stderr
        return
    check(N, K, H, F, E, capacity)
    check_status(torch.device("cuda", torch.cuda.current_device()))


def check(N, K, H, F, E, capacity):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF

    g = torch.Generator(device="cuda").manual_seed(N + F)
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).to(torch.bfloat16)
    idx = (torch.rand(N, E, device="cuda", generator=g) + torch.arange(E, device="cuda") * 0.05).topk(K, 1).indices
    gate = torch.rand(N, K, device="cuda", generator=g).requires_grad_()
    x, w13, w2, dy = mk(N, H), mk(E, 2 * F, H, scale=H ** -0.5), mk(E, H, F, scale=F ** -0.5), mk(N, H)
    y = OF.local_moe(x, gate, idx, w13, w2, capacity)
    y.backward(dy)
    drop = OF.capacity_drop_mask_reference(idx, E, capacity) if capacity else torch.zeros_like(idx, dtype=torch.bool)
    assert capacity == 0 or bool(drop.any())
    want = torch.zeros(N, K, dtype=torch.float64, device="cuda")
    out = torch.zeros(N, H, dtype=torch.float64, device="cuda")
    for e in range(E):
        t, k = ((idx == e) & ~drop).nonzero(as_tuple=True)
        # gate and up are kept in bf16 between the passes
        gu = (x[t].double() @ w13[e].double().t()).to(torch.bfloat16).double()
        h = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
        want[t, k] = ((dy[t].double() @ w2[e].double()) * h).sum(1)
        out.index_add_(0, t, gate.detach().double()[t, k, None] * (h @ w2[e].double().t()))
    # The gradient is summed in fp32 from values that agree but for gate / up values near the middle between two bf16
    # ones, about one in a thousand, which may round the other way (4e-3 each): sqrt(1e-3) * 4e-3 = 1.3e-4.
    assert float((gate.grad.double() - want).norm()) <= 5e-4 * float(want.norm())
    # h, the result rows and their sum are rounded to bf16 (2^-9 at most each, a third of that on average)
    assert float((y.double() - out).norm()) <= 5e-3 * float(out.norm())
