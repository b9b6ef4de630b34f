"""Few rows per expert: the tiles of 256, 128 and 64 rows of weights that fill the SMs give the bits of full tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,N,H,F", [
    (64, 200, 512, 1024),   # 128 rows of weights in the first GEMM, 256 in the second
    (16, 60, 1024, 512),    # 128 and 64
    (8, 100, 1032, 264),    # ragged columns of both
    (8, 1, 2048, 72),       # one row, a tile that is mostly past the edge
    (4, 250, 136, 200),     # several pieces of rows
    (148, 148, 256, 128),   # whole rounds with full tiles
])
def test_streamed_tiles_match_full_tiles(E, N, H, F):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops.kernels import check_status

    g = torch.Generator(device="cuda").manual_seed(E + N)
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).to(torch.bfloat16)
    idx = torch.randint(0, E, (N, 1), device="cuda", generator=g)
    x, w13, w2 = mk(N, H), mk(E, 2 * F, H, scale=H ** -0.5), mk(E, H, F, scale=F ** -0.5)
    gate = torch.rand(N, 1, device="cuda", generator=g) + 0.5
    want = OF.local_moe(x.clone().requires_grad_(), gate, idx, w13, w2).detach()  # full tiles
    with torch.no_grad():
        got = OF.local_moe(x, gate, idx, w13, w2)
    assert torch.equal(got, want)
    ref = OF.experts_reference(x.double(), idx, gate.double(), w13.double(), w2.double())
    assert float((got.double() - ref).norm()) <= 1e-2 * float(ref.norm())  # bf16 gate|up, h and result
    check_status(x.device)
