"""The expert layer without a backward pass, where padding rows are neither filled nor, with few rows per expert, loaded or
stored: the same bits as the forward that keeps everything, with the freed memory around it full of NaN."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,H,F", [
    ([1], 64, 72),                               # one row
    ([0, 32, 33, 64, 31, 0, 2, 96], 256, 136),   # edges of the 32-row pieces, empty experts
    ([97, 128, 1, 1, 1, 1, 1, 129], 1032, 320),  # a full tile and a second one among short ones; ragged K and N
    ([200, 60, 65, 3], 512, 256),                # more than 64 rows per expert: whole tiles, padding not filled
])
def test_inference_matches_the_training_forward(rows, H, F):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops.kernels import check_status

    torch.manual_seed(sum(rows))
    E, N = len(rows), sum(rows)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(N)].cuda()[:, None]
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda") * scale).to(torch.bfloat16)
    x, w13, w2 = mk(N, H), mk(E, 2 * F, H, scale=H ** -0.5), mk(E, H, F, scale=F ** -0.5)
    gate = torch.rand(N, 1, device="cuda") + 0.5
    want = OF.local_moe(x.clone().requires_grad_(), gate, idx, w13, w2).detach()
    for _ in range(3):
        junk = [torch.full((n,), float("nan"), device="cuda") for n in (1 << 22, 1 << 20, 1 << 18, 1 << 16)]
        del junk
        with torch.no_grad():
            got = OF.local_moe(x, gate, idx, w13, w2)
        assert torch.equal(got, want)
    check_status(x.device)
