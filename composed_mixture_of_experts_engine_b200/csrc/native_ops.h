// Native layer operations that the autograd nodes in bindings_autograd.cpp are made of; each is defined in the binding file
// of its part of the package.
#pragma once
#include <torch/extension.h>

#include <optional>
#include <tuple>

namespace cmoe {

using OptTensor = std::optional<torch::Tensor>;

// bindings_router.cpp.  (idx32, w32, idx64, w16, logits, lse, counts, counts64, mean_prob, stats)
using RouteResult = std::tuple<OptTensor, OptTensor, torch::Tensor, torch::Tensor, OptTensor, OptTensor, OptTensor,
                               OptTensor, OptTensor, OptTensor>;
RouteResult router_route(const torch::Tensor& X, const torch::Tensor& Wg, int64_t K, bool full, const OptTensor& status);
std::tuple<OptTensor, OptTensor> router_grad(const torch::Tensor& X, const torch::Tensor& Wg, const torch::Tensor& logits,
                                             const torch::Tensor& lse, const torch::Tensor& idx32,
                                             const torch::Tensor& counts, const OptTensor& grad_w32,
                                             const OptTensor& grad_w16, const OptTensor& grad_aux, const OptTensor& grad_z,
                                             bool need_tokens, bool need_gate, bool gate_bf16, const OptTensor& status);

// bindings_moe.cpp.  (y, plan, xp, hact, gu, yp) and (dx, d_gate, dw13, dw2)
using MoeForward = std::tuple<torch::Tensor, torch::Tensor, OptTensor, OptTensor, OptTensor, OptTensor>;
MoeForward moe_local_forward(const torch::Tensor& x, const torch::Tensor& gate_w32, const torch::Tensor& idx32,
                             const torch::Tensor& w13, const torch::Tensor& w2, int64_t capacity, bool keep,
                             const OptTensor& status, const OptTensor& overflow, const OptTensor& made_plan);
using MoeBackward = std::tuple<OptTensor, OptTensor, OptTensor, OptTensor>;
MoeBackward moe_local_backward(const torch::Tensor& dy, const torch::Tensor& plan, const torch::Tensor& xp,
                               const torch::Tensor& hact, const torch::Tensor& gu, const torch::Tensor& yp,
                               const torch::Tensor& gate_w32, const torch::Tensor& w13, const torch::Tensor& w2,
                               bool need_dx, bool need_gate, const OptTensor& main13, const OptTensor& main2,
                               const OptTensor& status);

// bindings.cpp
std::tuple<torch::Tensor, torch::Tensor, torch::Tensor> add_rmsnorm(const torch::Tensor& x, const OptTensor& delta,
                                                                    const torch::Tensor& w, double eps);
std::tuple<torch::Tensor, OptTensor> add_rmsnorm_grad(const torch::Tensor& dy, const OptTensor& dsum,
                                                      const torch::Tensor& x, const torch::Tensor& w,
                                                      const torch::Tensor& rstd, bool need_dw, const OptTensor& main);
void rope(torch::Tensor& t, const torch::Tensor& cos_tab, const torch::Tensor& sin_tab, int64_t seq, bool inverse);
void qkv_grad_pack(const torch::Tensor& dq, const torch::Tensor& dk, const torch::Tensor& dv, torch::Tensor& out,
                   const torch::Tensor& cos_tab, const torch::Tensor& sin_tab);

}  // namespace cmoe
