#include "host_ops.h"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "ops.cuh"

namespace cmoe {

using torch::Tensor;

namespace {

void check(cudaError_t e, const char* what) {
  TORCH_CHECK(e == cudaSuccess, "cmoe: ", what, " failed: ", cudaGetErrorString(e));
}
void check_bf16_matrix(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.stride(1) == 1, name,
              " must be a CUDA bf16 matrix with unit inner stride");
}
GemmArgs operands(const Tensor& A, bool a_mn, const Tensor& B, bool b_mn) {
  check_bf16_matrix(A, "A");
  check_bf16_matrix(B, "B");
  GemmArgs g;
  g.A = A.data_ptr();
  g.a_rows = A.size(0);
  g.a_cols = A.size(1);
  g.a_ld = A.stride(0);
  g.a_mn = a_mn;
  g.B = B.data_ptr();
  g.b_rows = B.size(0);
  g.b_cols = B.size(1);
  g.b_ld = B.stride(0);
  g.b_mn = b_mn;
  g.num_sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  return g;
}
bool two_cta() {
  static const bool on = [] {
    const char* v = std::getenv("CMOE_GEMM_2CTA");
    return v == nullptr || (v[0] != '\0' && v[0] != '0');
  }();
  return on;
}
// `stats`, where given: takes the softmax statistics of the rows
Tensor dense(const Tensor& x, const Tensor& w, bool b_mn, Tensor out, int* status, Tensor* stats = nullptr) {
  const c10::cuda::CUDAGuard guard(x.device());
  GemmArgs g = operands(x, false, w, b_mn);
  const int64_t M = x.size(0), N = w.size(b_mn ? 1 : 0), K = x.size(1);
  TORCH_CHECK(w.size(b_mn ? 0 : 1) == K, "dense GEMM: inner sizes differ");
  if (!out.defined()) out = at::empty({M, N}, x.options());
  check_bf16_matrix(out, "out");
  g.M = static_cast<int>(M);
  g.N = static_cast<int>(N);
  g.K = static_cast<int>(K);
  g.D = out.data_ptr();
  g.ldd = out.stride(0);
  g.status = status;
  if (stats != nullptr && two_cta() && gemm_2cta_supported(g)) {
    *stats = at::empty({M, (N + 255) / 256, 2}, x.options().dtype(at::kFloat));
    g.row_stats = reinterpret_cast<float2*>(stats->data_ptr<float>());
  }
  launch_gemm_any(g, at::cuda::getCurrentCUDAStream().stream());
  return out;
}

// Into how many pieces the contraction over R rows of an M x N weight gradient is cut.  The two-SM kernel works on
// 256 x 256 tiles, one per pair of SMs, 0.4 us per 64 rows of a tile; pieces fill the SMs that a small output leaves
// idle, but each costs a write and a read of the output in fp32 (8 bytes an element at about 5 bytes a picosecond)
// and a further launch.  Least estimated time wins, so 1 for large outputs and short contractions.
int wgrad_pieces(int64_t R, int64_t M, int64_t N, int sms) {
  const double pairs = sms / 2, tiles = double((M + 255) / 256) * double((N + 255) / 256);
  const int64_t blocks = (R + 63) / 64;
  int best = 1;
  double best_us = 0;
  for (int s = 1; s <= 16 && (s == 1 || blocks >= 8 * s); ++s) {
    const double waves = std::max(1.0, std::ceil(tiles * s / pairs));
    const double us = waves * (double((blocks + s - 1) / s) * 0.4 + 2.0) + (s > 1 ? s * double(M * N) * 8e-6 / 5.0 + 3.0 : 0.0);
    if (s == 1 || us < 0.95 * best_us) {
      best = s;
      best_us = us;
    }
  }
  return best;
}

}  // namespace

Tensor contiguous_aligned(const Tensor& t) {
  if (!t.is_contiguous()) return t.contiguous();
  return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone();
}

void launch_gemm_any(const GemmArgs& g, cudaStream_t stream) {
  if (two_cta() && gemm_2cta_supported(g))
    check(launch_gemm_2cta(g, stream), "launch_gemm_2cta");
  else
    check(launch_gemm(g, stream), "launch_gemm");
}

Tensor dense_nt(const Tensor& x, const Tensor& w, Tensor out, int* status) { return dense(x, w, false, out, status); }
std::pair<Tensor, Tensor> dense_nt_stats(const Tensor& x, const Tensor& w, int* status) {
  Tensor stats;
  Tensor y = dense(x, w, false, Tensor(), status, &stats);
  return {y, stats};
}
Tensor dense_nn(const Tensor& x, const Tensor& w, Tensor out, int* status) { return dense(x, w, true, out, status); }

void dense_wgrad(const Tensor& a, const Tensor& b, Tensor& out, bool accumulate, int* status, int64_t want_pieces) {
  const c10::cuda::CUDAGuard guard(a.device());
  GemmArgs g = operands(a, true, b, true);
  const int64_t R = a.size(0), M = a.size(1), N = b.size(1);
  const bool fp32 = out.scalar_type() == at::kFloat;
  TORCH_CHECK(b.size(0) == R && out.dim() == 2 && out.size(0) == M && out.size(1) == N && out.stride(1) == 1 &&
                  (fp32 || (out.scalar_type() == at::kBFloat16 && !accumulate)),
              "wgrad: bad output");
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
  // every way of writing `out` uses 16-byte vectors, the sum of the pieces over all of it as one run
  TORCH_CHECK(reinterpret_cast<uintptr_t>(out.data_ptr()) % 16 == 0 && out.stride(0) * (fp32 ? 4 : 2) % 16 == 0,
              "wgrad: the rows of the output must start on 16-byte boundaries");
  int pieces = 1;
  if (out.is_contiguous() && (M * N) % 4 == 0)
    pieces = want_pieces > 0 ? static_cast<int>(want_pieces) : wgrad_pieces(R, M, N, g.num_sms);
  const int64_t chunk = ((R + pieces - 1) / pieces + 63) / 64 * 64;
  g.mode = GEMM_GROUPED_K;
  g.M = static_cast<int>(M);
  g.N = static_cast<int>(N);
  g.groups = pieces;
  g.k_chunk = static_cast<int>(chunk);
  g.d_group_stride = M * N;
  g.ldd = pieces > 1 ? N : out.stride(0);
  g.status = status;
  Tensor part;
  if (pieces > 1) {
    part = at::empty({pieces, M, N}, a.options().dtype(at::kFloat));
    g.D = part.data_ptr();
    g.d_fp32 = 1;
  } else {
    g.D = out.data_ptr();
    g.d_fp32 = fp32;
    g.accumulate = accumulate;
  }
  launch_gemm_any(g, stream);
  if (pieces > 1)
    check(launch_splitk_reduce(part.data_ptr<float>(), pieces, M * N, out.data_ptr(), !fp32, accumulate, stream),
          "splitk_reduce");
}

}  // namespace cmoe
