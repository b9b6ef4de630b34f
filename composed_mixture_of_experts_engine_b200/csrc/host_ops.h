// Native host building blocks shared by the binding files: GEMM launches on tensors, without Python in between.
#pragma once
#include <torch/extension.h>

#include "gemm.cuh"

namespace cmoe {

// `t`, or a contiguous copy on a 16-byte boundary where it is not that already (saved tensors may come back from a hook in
// any layout)
torch::Tensor contiguous_aligned(const torch::Tensor& t);

// Launches `g` on the two-SM kernel where it qualifies (CMOE_GEMM_2CTA=0: never), on the one-CTA kernel otherwise.
void launch_gemm_any(const GemmArgs& g, cudaStream_t stream);

// y[M, N] = x[M, K] @ w[N, K]^T (out: bf16, allocated when undefined)
torch::Tensor dense_nt(const torch::Tensor& x, const torch::Tensor& w, torch::Tensor out, int* status);
// the same with the softmax statistics of the rows (GemmArgs::row_stats, fp32 [M, ceil(N / 256), 2]) where the kernel that
// runs can leave them; undefined otherwise
std::pair<torch::Tensor, torch::Tensor> dense_nt_stats(const torch::Tensor& x, const torch::Tensor& w, int* status);
// y[M, K] = x[M, N] @ w[N, K]
torch::Tensor dense_nn(const torch::Tensor& x, const torch::Tensor& w, torch::Tensor out, int* status);
// out[M, N] (+)= a[R, M]^T @ b[R, N]; out fp32 (stored, or added to) or bf16 (stored), its rows on 16-byte
// boundaries.  The contraction is cut into `pieces` (0: as many as are worth it) that run side by side where out is contiguous.
void dense_wgrad(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& out, bool accumulate, int* status,
                 int64_t pieces = 0);

}  // namespace cmoe
