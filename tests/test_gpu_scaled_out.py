"""The scaled output stores or adds as its caller says, not as the output's type suggests."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 1020, 4100])
def test_store_and_add_follow_the_flag(n):
    from composed_mixture_of_experts_engine_b200.ops import _ext

    torch.manual_seed(n)
    x, s = torch.randn(n, device="cuda"), torch.tensor([0.37], device="cuda")
    out = torch.full((n,), float("nan"), device="cuda")
    _ext.ext().scaled_out(x, s, out, False)  # memory that nobody has written to must not be read
    assert torch.equal(out, x * s)
    _ext.ext().scaled_out(x, s, out, True)
    assert torch.allclose(out.double(), 2 * float(s) * x.double(), rtol=2.0 ** -22, atol=0)
    half = torch.zeros(n, device="cuda", dtype=torch.bfloat16)
    _ext.ext().scaled_out(x, s, half, False)
    assert torch.equal(half, (x * s).to(torch.bfloat16))
    with pytest.raises(RuntimeError):
        _ext.ext().scaled_out(x, s, half, True)
