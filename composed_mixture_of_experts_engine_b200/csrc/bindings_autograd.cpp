// Autograd nodes of the layer operations, forward and backward without Python: a training step of small layers is bound by
// its host work, and a Python autograd function costs 30 to 75 us per direction on the host that feeds a B200 (argument
// checks, context, tensor constructions, the interpreter lock in the backward thread), several times what its kernels take.
//
// Each node does what the Python function of the same operation does (ops/functional.py, ops/moe_router.py); those stay for
// what only they serve: traces, which record them by name, and forward-mode tangents, which they refuse.
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include "host_ops.h"
#include "native_ops.h"

namespace {

using cmoe::OptTensor;
using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

// tensors that are no inputs of a node: passed by value, so that the node does not take them for some
struct Aside {
  Tensor a, b;
};

OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }
Tensor or_none(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

// `weight.main_grad`, the fp32 buffer that the optimizer gave the parameter, as it is when the gradient is made
OptTensor main_grad(const Tensor& weight) {
  const pybind11::gil_scoped_acquire gil;
  const auto o = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(weight));
  if (!pybind11::hasattr(o, "main_grad")) return std::nullopt;
  const pybind11::object m = o.attr("main_grad");
  return m.is_none() ? OptTensor() : OptTensor(m.cast<Tensor>());
}

// The same for a norm's weight, where its gradient may go straight into that buffer: one that the kernel can add to, while
// nobody waits for the gradient itself - no hook on the weight or on the node that accumulates its gradient, no call that
// asks for the gradients of given tensors.  Elsewhere autograd gets it, and the optimizer adds what is in `.grad` later.
OptTensor norm_main_grad(const Tensor& weight) {
  const OptTensor main = main_grad(weight);
  if (!main.has_value() || !weight.is_leaf() || main->scalar_type() != at::kFloat || !main->is_contiguous() ||
      main->numel() != weight.numel() || main->device() != weight.device())
    return std::nullopt;
  const auto* asked_for = torch::autograd::get_current_graph_task_exec_info();
  if (asked_for != nullptr && !asked_for->empty()) return std::nullopt;
  if (!torch::autograd::impl::hooks(weight).empty() || torch::autograd::impl::post_acc_grad_hooks(weight) != nullptr)
    return std::nullopt;
  const auto node = torch::autograd::impl::try_get_grad_accumulator(weight);
  if (node != nullptr && !(node->pre_hooks().empty() && node->post_hooks().empty())) return std::nullopt;
  return main;
}

// ---- y = x @ weight^T -------------------------------------------------------------------------------------------
struct LinearFn : Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Aside& status) {
    const Tensor x2 = cmoe::contiguous_aligned(x.reshape({-1, x.size(-1)}));
    auto sizes = x.sizes().vec();
    sizes.back() = weight.size(0);
    Tensor y = at::empty(sizes, x.options());
    cmoe::dense_nt(x2, weight, y.view({-1, weight.size(0)}), status.a.data_ptr<int>());
    ctx->save_for_backward({x2, weight});
    ctx->saved_data["status"] = status.a;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor x2 = cmoe::contiguous_aligned(saved[0]), &weight = saved[1];
    const Tensor status = ctx->saved_data["status"].toTensor();
    int* st = status.data_ptr<int>();
    const int64_t N = weight.size(0), K = weight.size(1);
    const Tensor dy2 = cmoe::contiguous_aligned(grads[0].reshape({-1, N}));
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) {
      auto sizes = grads[0].sizes().vec();
      sizes.back() = K;
      dx = at::empty(sizes, dy2.options());
      cmoe::dense_nn(dy2, weight, dx.view({-1, K}), st);
    }
    if (ctx->needs_input_grad(1)) {
      if (OptTensor main = main_grad(weight)) {
        if (main->scalar_type() == at::kFloat && main->is_contiguous() && main->dim() == 2 && K % 4 == 0 &&
            reinterpret_cast<uintptr_t>(main->data_ptr()) % 16 == 0) {
          cmoe::dense_wgrad(dy2, x2, *main, true, st);
        } else {  // a buffer that the kernels cannot add to
          Tensor res = at::empty({N, K}, dy2.options().dtype(at::kFloat));
          cmoe::dense_wgrad(dy2, x2, res, false, st);
          main->add_(res.to(main->scalar_type()));
        }
      } else {
        dw = at::empty({N, K}, weight.options());
        cmoe::dense_wgrad(dy2, x2, dw, false, st);
      }
    }
    return {dx, dw, Tensor()};
  }
};

// ---- (x + delta, norm of it) ------------------------------------------------------------------------------------
struct AddRMSNormFn : Function<AddRMSNormFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& delta, const Tensor& weight,
                               double eps) {
    auto [s, y, rstd] = cmoe::add_rmsnorm(x, delta, weight, eps);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({s, weight, rstd});
    ctx->saved_data["delta"] = delta.has_value();
    return {s, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    Tensor dx = grads[0], dw;
    if (grads[1].defined()) {
      // (counted over the tensors that the call was given)
      const bool need_dw = ctx->needs_input_grad(ctx->saved_data["delta"].toBool() ? 2 : 1);
      auto [d, w] = cmoe::add_rmsnorm_grad(grads[1], opt(grads[0]), saved[0], saved[1], saved[2], need_dw,
                                           need_dw ? norm_main_grad(saved[1]) : OptTensor());
      dx = d;
      dw = or_none(w);
    }
    return {dx, ctx->saved_data["delta"].toBool() ? dx : Tensor(), dw, Tensor()};
  }
};

// ---- RoPE on q and k and causal attention on the packed projection, as many k / v heads as q heads --------------------
struct RopeAttentionFn : Function<RopeAttentionFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Aside& tables, int64_t nh) {
    const int64_t B = qkv.size(0), S = qkv.size(1), heads = qkv.size(2), hd = qkv.size(3);
    const Tensor t = qkv.detach();
    Tensor rotated = t.view({B * S, heads, hd}).narrow(1, 0, 2 * nh);
    cmoe::rope(rotated, tables.a, tables.b, S, false);
    Tensor q, k, v, out;
    {
      const at::AutoGradMode on(true);
      q = t.narrow(2, 0, nh).permute({0, 2, 1, 3}).requires_grad_();
      k = t.narrow(2, nh, nh).permute({0, 2, 1, 3}).requires_grad_();
      v = t.narrow(2, 2 * nh, nh).permute({0, 2, 1, 3}).requires_grad_();
      out = at::scaled_dot_product_attention(q, k, v, {}, 0.0, true);
    }
    ctx->saved_data["inner"] = c10::List<Tensor>({q, k, v, out});
    ctx->save_for_backward({tables.a, tables.b});
    return out.detach().permute({0, 2, 1, 3}).contiguous();
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto it = ctx->saved_data.find("inner");
    TORCH_CHECK(it != ctx->saved_data.end(), "the attention's inner graph has been used by an earlier backward pass");
    const auto inner = it->second.toTensorVector();
    ctx->saved_data.erase(it);
    const auto g = torch::autograd::grad({inner[3]}, {inner[0], inner[1], inner[2]}, {grads[0].permute({0, 2, 1, 3})});
    const int64_t nh = inner[0].size(1), S = inner[0].size(2), hd = inner[0].size(3), B = inner[0].size(0);
    Tensor dqkv = at::empty({B, S, 3 * nh, hd}, grads[0].options());
    bool vectors = true;
    for (const Tensor& t : g)
      vectors = vectors && t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0;
    if (vectors) {
      cmoe::qkv_grad_pack(g[0], g[1], g[2], dqkv, saved[0], saved[1]);
    } else {
      for (int i = 0; i < 3; ++i) dqkv.narrow(2, i * nh, nh).copy_(g[i].permute({0, 2, 1, 3}));
      Tensor rotated = dqkv.view({B * S, 3 * nh, hd}).narrow(1, 0, 2 * nh);
      cmoe::rope(rotated, saved[0], saved[1], S, true);
    }
    return {dqkv, Tensor(), Tensor()};
  }
};

// ---- router -----------------------------------------------------------------------------------------------------
// what a routing call leaves besides the node's outputs
struct RouterSide {
  OptTensor logits, lse, counts, counts64, mean_prob, stats;
};
struct RouterFn : Function<RouterFn> {
  // (w32, w16, aux, z, idx32, idx64)
  static variable_list forward(AutogradContext* ctx, const Tensor& tokens, const Tensor& gate_w, int64_t k,
                               const Aside& status, RouterSide* side) {
    auto [idx32, w32, idx64, w16, logits, lse, counts, counts64, mean_prob, stats] =
        cmoe::router_route(tokens, gate_w, k, true, status.a);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({tokens, gate_w, *logits, *lse, *idx32, *counts});
    ctx->saved_data["status"] = status.a;
    ctx->mark_non_differentiable({*idx32, idx64});
    *side = RouterSide{logits, lse, counts, counts64, mean_prob, stats};
    return {*w32, w16, stats->select(0, 0), stats->select(0, 1), *idx32, idx64};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    auto [gt, gg] = cmoe::router_grad(s[0], s[1], s[2], s[3], s[4], s[5], opt(g[0]), opt(g[1]), opt(g[2]), opt(g[3]),
                                      ctx->needs_input_grad(0), ctx->needs_input_grad(1), true,
                                      ctx->saved_data["status"].toTensor());
    return {or_none(gt), or_none(gg), Tensor(), Tensor(), Tensor()};
  }
};

// ---- expert layer -----------------------------------------------------------------------------------------------
struct MoEFn : Function<MoEFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate_w32, const Tensor& w13, const Tensor& w2,
                        const Aside& idx32_status, const OptTensor* made_plan, const OptTensor* overflow, int64_t capacity,
                        Tensor* plan_out) {
    auto [y, plan, xp, hact, gu, yp] = cmoe::moe_local_forward(x, gate_w32, idx32_status.a, w13, w2, capacity, true,
                                                               idx32_status.b, *overflow, *made_plan);
    ctx->save_for_backward({plan, or_none(xp), or_none(hact), or_none(gu), or_none(yp), gate_w32, w13, w2});
    ctx->saved_data["status"] = idx32_status.b;
    *plan_out = plan;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    auto [dx, d_gate, dw13, dw2] = cmoe::moe_local_backward(
        cmoe::contiguous_aligned(g[0]), s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], ctx->needs_input_grad(0),
        ctx->needs_input_grad(1), main_grad(s[6]), main_grad(s[7]), ctx->saved_data["status"].toTensor());
    return {or_none(dx), or_none(d_gate), or_none(dw13), or_none(dw2), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

void register_autograd(pybind11::module_& m) {
  m.def("linear", [](const Tensor& x, const Tensor& weight, const Tensor& status) {
    const c10::cuda::CUDAGuard guard(x.device());
    return LinearFn::apply(x, weight, Aside{status, {}});
  });
  m.def("add_rmsnorm_node", [](const Tensor& x, const OptTensor& delta, const Tensor& weight, double eps) {
    auto out = AddRMSNormFn::apply(x, delta, weight, eps);
    return std::make_tuple(out[0], out[1]);
  });
  m.def("norm_main_grad", &norm_main_grad);
  m.def("rope_attention", [](const Tensor& qkv, const Tensor& cos_tab, const Tensor& sin_tab, int64_t nh) {
    const c10::cuda::CUDAGuard guard(qkv.device());
    TORCH_CHECK(qkv.dim() == 4 && qkv.is_contiguous() && qkv.size(2) == 3 * nh, "qkv must be contiguous [B, S, 3 nh, hd]");
    return RopeAttentionFn::apply(qkv, Aside{cos_tab, sin_tab}, nh);
  });
  // (idx32, w32, idx64, w16, logits, lse, counts, counts64, mean_prob, stats), aux loss, z loss
  m.def("router_node", [](const Tensor& tokens, const Tensor& gate_w, int64_t k, const Tensor& status) {
    RouterSide s;
    auto out = RouterFn::apply(tokens, gate_w, k, Aside{status, {}}, &s);
    return std::make_tuple(std::make_tuple(out[4], out[0], out[5], out[1], s.logits, s.lse, s.counts, s.counts64,
                                           s.mean_prob, s.stats),
                           out[2], out[3]);
  });
  // (y, plan)
  m.def("moe_local_node", [](const Tensor& x, const Tensor& gate_w32, const Tensor& idx32, const Tensor& w13,
                             const Tensor& w2, int64_t capacity, const Tensor& status, const OptTensor& overflow,
                             const OptTensor& made_plan) {
    Tensor plan;
    Tensor y = MoEFn::apply(x, gate_w32, w13, w2, Aside{idx32, status}, &made_plan, &overflow, capacity, &plan);
    return std::make_tuple(y, plan);
  });
}
