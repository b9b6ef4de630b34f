"""Weight-gradient contraction cut into row pieces (ordered sum of the partial results), and the d(logits) kernel at
its expert-count edges; against fp32 / fp64 restatements."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,M,N", [(65, 256, 8), (100, 128, 72), (4096, 1024, 1024), (8190, 4096, 256), (5000, 264, 40),
                                   (16384, 2048, 2048)])
def test_wgrad_pieces_match_fp32(R, M, N):
    from composed_mixture_of_experts_engine_b200.ops import kernels

    torch.manual_seed(R + N)
    a = torch.randn(R, M, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(R, N, device="cuda", dtype=torch.bfloat16)
    want = a.double().t() @ b.double()
    # fp32 sums of R products of unit variance: error of one sum below R * 2^-24 of its rms sqrt(R), times a few
    tol = 4e-6 * R ** 0.5

    def rel(x):
        return float((x.double() - want).norm() / want.norm())

    got = kernels.linear_tn(a, b)
    assert got.dtype == torch.float32 and rel(got) < tol
    assert torch.equal(got, kernels.linear_tn(a, b))  # same inputs, same bits
    assert rel(kernels.linear_tn_acc(a, b, torch.ones(M, N, device="cuda")) - 1.0) < tol
    assert torch.equal(kernels.linear_tn(a, b, out_dtype=torch.bfloat16), got.to(torch.bfloat16))


@pytest.mark.parametrize("N,E,K", [(1, 8, 1), (33, 24, 3), (130, 64, 8), (257, 136, 6), (1000, 256, 8)])
def test_router_dlogits_at_expert_count_edges(N, E, K):
    from composed_mixture_of_experts_engine_b200.ops import _ext

    torch.manual_seed(N + E)
    lg = torch.randn(N, E, device="cuda")
    lse = torch.logsumexp(lg, -1)
    idx = torch.topk(lg, K, -1).indices.to(torch.int32)
    counts = torch.bincount(idx.flatten().long(), minlength=E).to(torch.int32)
    gw, ga, gz = torch.randn(N, K, device="cuda"), torch.tensor([0.3], device="cuda"), torch.tensor([0.2], device="cuda")
    for use in (True, False):  # with and without the two loss terms
        gl, gl16 = torch.empty(N, E, device="cuda"), torch.empty(N, E, device="cuda", dtype=torch.bfloat16)
        _ext.ext().router_bwd(lg, lse, idx, gw, counts, ga if use else None, gz if use else None, gl16, gl)
        x = lg.double().requires_grad_()
        p = torch.softmax(x, -1)
        sel = p.gather(1, idx.long())
        loss = (sel / sel.sum(-1, keepdim=True) * gw).sum()
        if use:
            loss = loss + 0.3 * E * (counts.double() / (N * K) * p.mean(0)).sum() + 0.2 * (torch.logsumexp(x, -1) ** 2).mean()
        loss.backward()
        assert torch.allclose(gl.double(), x.grad, atol=2e-6, rtol=1e-4)
        assert torch.equal(gl16, gl.to(torch.bfloat16))
