"""What the native RMSNorm is asked with before anything is launched."""

import pytest
import torch


@pytest.mark.parametrize("shape", [(), (0,), (4, 0), (2, 3, 0)])
def test_rows_without_columns_are_refused(shape):
    """... by an error: the row count is a quotient by their number."""
    from composed_mixture_of_experts_engine_b200.ops import _ext

    x = torch.zeros(shape, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="rows must have columns"):
        _ext.ext().add_rmsnorm(x, None, torch.zeros(shape[-1:], dtype=torch.bfloat16), 1e-5)
