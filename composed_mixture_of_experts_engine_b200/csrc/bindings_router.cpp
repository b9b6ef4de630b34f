// Native host path of the router: one call allocates every output of a routing pass and launches the kernel, so that
// a small routing call costs one binding call instead of eight tensor constructions and three casts in Python.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <map>
#include <mutex>
#include <optional>
#include <tuple>
#include <utility>

#include "host_ops.h"
#include "native_ops.h"
#include "router.cuh"

namespace {

using cmoe::OptTensor;
using cmoe::RouteResult;
using torch::Tensor;

// Statistics workspace, zero between launches (the kernel leaves it so).  One per (device, stream): launches on one
// stream run in order, launches on two streams must not share the accumulators.  At most kMaxWorkspaces are kept
// (3 KiB each); further streams get a fresh zeroed one per call.  So does a call under capture: a graph may be replayed
// on any stream, before or beside others that were captured on the same one, and its memory and the zero fill belong to
// that graph alone.
constexpr size_t kMaxWorkspaces = 256;
Tensor router_workspace(const c10::Device& dev, cudaStream_t stream) {
  static std::mutex mu;
  // never destroyed: at exit the allocator may be gone before this table
  static auto& kept = *new std::map<std::pair<int, cudaStream_t>, Tensor>;
  const auto opt = at::TensorOptions().device(dev).dtype(at::kInt);
  const int64_t words = static_cast<int64_t>(cmoe::router_workspace_words(cmoe::kRouterMaxExperts));
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  const cudaError_t e = cudaStreamIsCapturing(stream, &capturing);
  TORCH_CHECK(e == cudaSuccess, "cmoe: cudaStreamIsCapturing failed: ", cudaGetErrorString(e));
  if (capturing != cudaStreamCaptureStatusNone) return at::zeros({words}, opt);
  const std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(static_cast<int>(dev.index()), stream);
  auto it = kept.find(key);
  if (it != kept.end()) return it->second;
  Tensor t = at::zeros({words}, opt);
  if (kept.size() < kMaxWorkspaces) kept.emplace(key, t);
  return t;
}

// (idx32, w32, idx64, w16, logits, lse, counts, counts64, mean_prob, stats).  `full` false: only the routing decision
// in its public types (idx64, w16) is produced, for callers that want no gradient and no statistics.
RouteResult router_route(const Tensor& X, const Tensor& Wg, int64_t K, bool full, const OptTensor& status) {
  TORCH_CHECK(X.is_cuda() && X.scalar_type() == at::kBFloat16 && X.dim() == 2 && X.stride(1) == 1,
              "X must be a CUDA bf16 matrix with unit inner stride");
  TORCH_CHECK(Wg.is_cuda() && Wg.scalar_type() == at::kBFloat16 && Wg.dim() == 2 && Wg.is_contiguous() &&
                  Wg.size(0) == X.size(1),
              "Wg must be contiguous bf16 [H, E]");
  const c10::cuda::CUDAGuard guard(X.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
  const int64_t N = X.size(0), E = Wg.size(1);
  const auto f32 = X.options().dtype(at::kFloat), i32 = X.options().dtype(at::kInt), i64 = X.options().dtype(at::kLong);
  cmoe::RouterFwdArgs a;
  a.X = X.data_ptr();
  a.n_tokens = N;
  a.H = static_cast<int>(X.size(1));
  a.ldx = X.stride(0);
  a.Wg = Wg.data_ptr();
  a.E = static_cast<int>(E);
  a.K = static_cast<int>(K);
  a.num_sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  Tensor idx64 = at::empty({N, K}, i64), w16 = at::empty({N, K}, X.options());
  a.topk_idx64 = reinterpret_cast<long long*>(idx64.data_ptr<int64_t>());
  a.topk_w_bf16 = w16.data_ptr();
  OptTensor idx32, w32, logits, lse, counts, counts64, mean_prob, stats;
  Tensor ws;
  if (full) {
    idx32 = at::empty({N, K}, i32);
    w32 = at::empty({N, K}, f32);
    logits = at::empty({N, E}, f32);
    lse = at::empty({N}, f32);
    counts = at::empty({E}, i32);
    counts64 = at::empty({E}, i64);
    mean_prob = at::empty({E}, f32);
    stats = at::empty({4}, f32);
    ws = router_workspace(X.device(), stream);
    a.topk_idx = idx32->data_ptr<int>();
    a.topk_w = w32->data_ptr<float>();
    a.logits = logits->data_ptr<float>();
    a.lse = lse->data_ptr<float>();
    a.counts = counts->data_ptr<int>();
    a.counts64 = reinterpret_cast<long long*>(counts64->data_ptr<int64_t>());
    a.mean_prob = mean_prob->data_ptr<float>();
    a.stats = stats->data_ptr<float>();
    a.workspace = reinterpret_cast<uint32_t*>(ws.data_ptr());
  }
  a.status = status.has_value() ? status->data_ptr<int>() : nullptr;
  const cudaError_t e = cmoe::launch_router_fwd(a, stream);
  TORCH_CHECK(e == cudaSuccess, "cmoe: launch_router_fwd failed: ", cudaGetErrorString(e));
  return {idx32, w32, idx64, w16, logits, lse, counts, counts64, mean_prob, stats};
}

// (grad_tokens, grad_gate) from the upstream gradients of the gate weights (fp32 and / or bf16 view of the same
// values), the load-balance loss and the z-loss: the d(logits) kernel, then the two contractions with it.
std::tuple<OptTensor, OptTensor> router_grad(const Tensor& X, const Tensor& Wg, const Tensor& logits_in, const Tensor& lse,
                                             const Tensor& idx32, const Tensor& counts_in, const OptTensor& grad_w32,
                                             const OptTensor& grad_w16, const OptTensor& grad_aux,
                                             const OptTensor& grad_z, bool need_tokens, bool need_gate, bool gate_bf16,
                                             const OptTensor& status) {
  const c10::cuda::CUDAGuard guard(X.device());
  const Tensor logits = cmoe::contiguous_aligned(logits_in), counts = cmoe::contiguous_aligned(counts_in);
  const auto as_f32 = [](const OptTensor& t) {
    return t.has_value() ? OptTensor(t->to(at::kFloat).contiguous()) : OptTensor();
  };
  OptTensor gw = as_f32(grad_w32);
  if (grad_w16.has_value()) gw = gw.has_value() ? (*gw + *grad_w16).contiguous() : as_f32(grad_w16);
  const OptTensor ga = as_f32(grad_aux), gz = as_f32(grad_z);
  Tensor gl = at::empty(logits.sizes(), X.options());
  cmoe::RouterBwdArgs a;
  a.logits = logits.data_ptr<float>();
  a.lse = lse.data_ptr<float>();
  a.topk_idx = idx32.data_ptr<int>();
  a.grad_w = gw.has_value() ? gw->data_ptr<float>() : nullptr;
  a.counts = counts.data_ptr<int>();
  a.grad_aux = ga.has_value() ? ga->data_ptr<float>() : nullptr;
  a.grad_z = gz.has_value() ? gz->data_ptr<float>() : nullptr;
  a.n_tokens = logits.size(0);
  a.E = static_cast<int>(logits.size(1));
  a.K = static_cast<int>(idx32.size(1));
  a.grad_logits_bf16 = gl.data_ptr();
  const cudaError_t e = cmoe::launch_router_bwd(a, at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "cmoe: launch_router_bwd failed: ", cudaGetErrorString(e));
  int* st = status.has_value() ? status->data_ptr<int>() : nullptr;
  std::tuple<OptTensor, OptTensor> out;
  if (need_tokens) std::get<0>(out) = cmoe::dense_nt(gl, Wg, Tensor(), st);  // [N, E] x [H, E]^T
  if (need_gate) {                                                          // tokens^T [H, N] x gl [N, E]
    Tensor g = at::empty({X.size(1), gl.size(1)}, gate_bf16 ? X.options() : X.options().dtype(at::kFloat));
    cmoe::dense_wgrad(X, gl, g, false, st);
    std::get<1>(out) = g;
  }
  return out;
}

}  // namespace

namespace cmoe {
RouteResult router_route(const Tensor& X, const Tensor& Wg, int64_t K, bool full, const OptTensor& status) {
  return ::router_route(X, Wg, K, full, status);
}
std::tuple<OptTensor, OptTensor> router_grad(const Tensor& X, const Tensor& Wg, const Tensor& logits, const Tensor& lse,
                                             const Tensor& idx32, const Tensor& counts, const OptTensor& grad_w32,
                                             const OptTensor& grad_w16, const OptTensor& grad_aux, const OptTensor& grad_z,
                                             bool need_tokens, bool need_gate, bool gate_bf16, const OptTensor& status) {
  return ::router_grad(X, Wg, logits, lse, idx32, counts, grad_w32, grad_w16, grad_aux, grad_z, need_tokens, need_gate,
                       gate_bf16, status);
}
}  // namespace cmoe

void register_router(pybind11::module_& m) {
  m.def("router_route", &router_route);
  m.def("router_grad", &router_grad);
}
