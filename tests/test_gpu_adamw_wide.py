"""The update in 32-byte accesses against the one for any other form: the same bits; and at the edges of its launch shape."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 2040, 2048, 2056, 1 << 20])
@pytest.mark.parametrize("zero", [True, False])
def test_wide_update_has_the_bits_of_the_other(n, zero):
    from composed_mixture_of_experts_engine_b200.ops import _ext

    g = torch.Generator(device="cuda").manual_seed(n)
    base = [torch.randn(n + 8, device="cuda", generator=g) for _ in range(4)]
    base[2].abs_()
    ss = torch.tensor([9.0], device="cuda")
    results = []
    for off in (0, 4):  # 32-byte boundaries, 16-byte boundaries only
        p, m, v, grad = (torch.empty(n + 8, device="cuda")[off:off + n].copy_(t[:n]) for t in base)
        p16 = torch.empty(n + 8, device="cuda", dtype=torch.bfloat16)[2 * off:2 * off + n]
        assert (p.data_ptr() % 32 == 0) == (off == 0)
        _ext.ext().adamw(p, p16, m, v, grad, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, 0.5, 1.0, ss, zero)
        results.append((p, p16, m, v, grad))
        assert torch.equal(p16, p.to(torch.bfloat16))
        assert (float(grad.abs().max()) == 0.0) if zero else torch.equal(grad, base[3][:n])
    for a, b in zip(*results):
        assert torch.equal(a, b)
