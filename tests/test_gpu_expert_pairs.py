"""The expert layer where its grouped GEMMs run on pairs of SMs: experts with odd and even numbers of 128-row tiles, one
tile, none, and widths that fill no tile, forward and backward, against float64 autograd."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,H,F,main_grad", [
    ([128, 129, 385], 256, 136, False),       # one tile, a pair, two pairs; F one piece past a tile
    ([0, 256, 0, 300, 1], 64, 72, True),      # empty experts, a single row; K of one block
    ([3000, 1], 192, 1000, False),            # many pairs next to one row
    ([640, 513, 2000, 90], 1032, 320, True),  # K and N that end inside a block
])
def test_layer_on_pairs_matches_float64(rows, H, F, main_grad):
    from composed_mixture_of_experts_engine_b200.ops import functional as OF
    from composed_mixture_of_experts_engine_b200.ops.kernels import check_status

    torch.manual_seed(sum(rows))
    E, N = len(rows), sum(rows)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(N)].cuda()[:, None]
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda") * scale).to(torch.bfloat16)
    x, w13, w2, dy = mk(N, H), mk(E, 2 * F, H, scale=H ** -0.5), mk(E, H, F, scale=F ** -0.5), mk(N, H)
    gate = torch.rand(N, 1, device="cuda") + 0.5
    want_in = [t.double().requires_grad_() for t in (x, gate, w13, w2)]
    xd, gd, w13d, w2d = want_in
    want = torch.zeros(N, H, device="cuda", dtype=torch.float64)
    for e in range(E):
        tok = (idx[:, 0] == e).nonzero()[:, 0]
        gu = xd[tok] @ w13d[e].t()
        want = want.index_add(0, tok, (torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]) @ w2d[e].t() * gd[tok])
    want.backward(dy.double())
    got_in = [t.clone().requires_grad_() for t in (x, gate, w13, w2)]
    if main_grad:
        for p in got_in[2:]:
            p.main_grad = torch.zeros(p.shape, device="cuda")
    got = OF.local_moe(got_in[0], got_in[1], idx, got_in[2], got_in[3])
    got.backward(dy)
    check_status(x.device)
    pairs = [(got, want)] + [(g.main_grad if main_grad and i > 1 else g.grad, w.grad)
                             for i, (g, w) in enumerate(zip(got_in, want_in))]
    # a rounding to bf16 has a relative error of 2^-9 / sqrt(3) (root mean square); at most seven of them lie between the
    # inputs and any result: 3e-3, doubled
    for g, w in pairs:
        assert float((g.double() - w).norm()) <= 6e-3 * float(w.norm())
