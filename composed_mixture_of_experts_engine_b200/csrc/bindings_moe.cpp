// Native host path of the expert layer on one GPU: row plan -> gather -> grouped SwiGLU GEMMs -> weighted combine, and
// its backward, each as one binding call that allocates and launches everything.  A layer call of a few hundred
// tokens is bound by its host work: fourteen tensor constructions, six binding calls and their argument checks took
// longer in Python than the kernels on the GPU.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <optional>
#include <string>
#include <tuple>

#include "host_ops.h"
#include "native_ops.h"
#include "ops.cuh"

namespace {

using cmoe::OptTensor;
using Forward = cmoe::MoeForward;
using Backward = cmoe::MoeBackward;
using torch::Tensor;

void check(cudaError_t e, const char* what) {
  TORCH_CHECK(e == cudaSuccess, "cmoe: ", what, " failed: ", cudaGetErrorString(e));
}
int* status_ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr<int>() : nullptr; }

// The tables of a row plan in one int32 buffer (see MoePlanArgs in ops.cuh for their meaning).
struct PlanTables {
  int64_t n_slots, cap_rows, E;
  int64_t row_slot, group_offsets, tile_group, pair_tile, num_pairs, tile_rows, group_order, num_m_tiles, counts_kept, words;  // offsets; slot_row is at 0
  PlanTables(int64_t n_slots_, int64_t E_) : n_slots(n_slots_), E(E_) {
    // worst case of the padded layout: every slot kept, up to 127 padding rows for every expert that has a slot
    cap_rows = (n_slots + std::min(E, n_slots) * 127 + 127) / 128 * 128;
    row_slot = n_slots;
    group_offsets = row_slot + cap_rows;
    tile_group = group_offsets + E + 1;
    pair_tile = tile_group + cap_rows / 128;
    num_pairs = pair_tile + cap_rows / 128;
    tile_rows = num_pairs + 1;
    group_order = tile_rows + cap_rows / 128;
    num_m_tiles = group_order + E;
    counts_kept = num_m_tiles + 1;
    words = counts_kept + E;
  }
};

// the row kernels read and write rows in 16-byte vectors
void check_rows(const Tensor& t, const char* name) {
  TORCH_CHECK(reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && (t.size(0) <= 1 || t.stride(0) % 8 == 0) &&
                  t.size(1) % 8 == 0,
              name, ": rows must be multiples of 8 columns and start on 16-byte boundaries");
}

struct Shapes {
  int64_t N, K, H, E, F;
};
Shapes check_shapes(const Tensor& x, const Tensor& idx32, const Tensor& w13, const Tensor& w2) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1,
              "x must be a CUDA bf16 matrix with unit inner stride");
  check_rows(x, "x");
  TORCH_CHECK(idx32.scalar_type() == at::kInt && idx32.dim() == 2 && idx32.is_contiguous() && idx32.size(0) == x.size(0),
              "idx must be contiguous int32 [N, K]");
  TORCH_CHECK(w13.scalar_type() == at::kBFloat16 && w13.dim() == 3 && w13.is_contiguous() && w13.size(2) == x.size(1) &&
                  w13.size(1) % 2 == 0,
              "w13 must be contiguous bf16 [E, 2F, H]");
  const Shapes s{x.size(0), idx32.size(1), x.size(1), w13.size(0), w13.size(1) / 2};
  TORCH_CHECK(w2.scalar_type() == at::kBFloat16 && w2.is_contiguous() && w2.dim() == 3 && w2.size(0) == s.E &&
                  w2.size(1) == s.H && w2.size(2) == s.F,
              "w2 must be contiguous bf16 [E, H, F]");
  return s;
}

// Rows of B in a tile where a layer of few rows streams its weights: the width with which nearly whole rounds of tiles
// fill the SMs, for what counts is that all of them load all the time.  64 rows only where wider tiles leave the chip
// half empty: a k-block of 8 KiB takes its threads as long to issue as one of 16.  GPU time of the layer with tiles of 256 /
// 128 / 64 rows in both GEMMs: 64 tokens top-8, E 64 H 2048 F 1024 (3.46 rounds of 256, 6.92 of 128) 170.2 / 162.3 / 196.5
// us, 5 tokens 99.4 / 91.2 / 107.3; 8 tokens top-2, E 8 H 4096 F 4096 154.7 / 160.9 / 188.7; 250 tokens top-2, E 16 H 1024 F
// 512 44.3 / 40.3 / 44.2.
int streamed_tile(int64_t m_tiles, int64_t N, int epilogue, int sms) {
  int best = 256;
  double best_fill = 0.0;
  for (int bn : {256, 128, 64}) {
    const int64_t cols = epilogue == cmoe::EPI_SWIGLU_FWD ? bn / 2 : bn;
    const double rounds = static_cast<double>(m_tiles * ((N + cols - 1) / cols)) / sms;
    const double fill = rounds / std::ceil(rounds) * (bn == 64 ? 0.75 : 1.0);
    if (fill > 1.05 * best_fill) {
      best = bn;
      best_fill = fill;
    }
  }
  return best;
}

// a grouped-by-rows launch over the tiles of `plan`: D[rows, N] = A[rows, K] * B (one [b_rows, b_cols] block per expert)
cmoe::GemmArgs grouped_rows(const Tensor& A, const Tensor& B, int64_t b_group_rows, bool b_mn, const Tensor& D, int64_t N,
                            int64_t K, const PlanTables& pt, int* plan, int* status,
                            int epilogue = cmoe::EPI_STORE, bool training = true, bool short_tiles = false) {
  cmoe::GemmArgs g;
  g.A = A.data_ptr();
  g.a_rows = A.size(0);
  g.a_cols = A.size(1);
  g.a_ld = A.stride(0);
  g.B = B.data_ptr();
  g.b_rows = pt.E * b_group_rows;
  g.b_cols = B.size(2);
  g.b_ld = B.size(2);
  g.b_mn = b_mn;
  g.mode = cmoe::GEMM_GROUPED_M;
  g.N = static_cast<int>(N);
  g.K = static_cast<int>(K);
  g.groups = static_cast<int>(pt.E);
  g.b_group_rows = b_group_rows;
  g.tile_group = plan + pt.tile_group;
  g.num_m_tiles = plan + pt.num_m_tiles;
  g.max_m_tiles = static_cast<int>(pt.cap_rows / 128);
  g.rows_per_group = pt.n_slots / pt.E;
  g.D = D.data_ptr();
  g.ldd = D.stride(0);
  g.status = status;
  g.num_sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  g.epilogue = epilogue;
  g.b_early = 1;  // weights and row plan are older than the kernel before each of these launches
  // One tile of most experts.  Whatever the size of the weights: in a model other layers' weights come before they are read
  // again.  Decoders of layers with 50 MB of weights (E 16 H 1024 F 512), kept / first to leave: one layer 300 tokens 101.2 /
  // 99.4 us, two 189.1 / 182.7, four 355.7 / 351.6, four at 16 tokens 309.5 / 296.2, training steps 0.1 % less.  Only a
  // single layer of 50 to 75 MB, called again and again, would find them in L2 (forward 46.1 / 46.5, 43.6 / 45.1; forward and
  // backward 134.7 / 136.5, 157.9 / 159.5); from 126 MB on it does not either (59.1 / 54.1 forward, 403 MB 103.5 / 98.8).
  g.b_once = g.rows_per_group <= 128;
  if (short_tiles) {
    g.tile_rows = plan + pt.tile_rows;
    g.tile_n = streamed_tile(std::min(pt.E, pt.n_slots), N, epilogue, g.num_sms);
    return g;
  }
  // Pairs of SMs on pairs of tiles, or single SMs on single tiles?  A pair needs about 0.85 of the time of a tile (it loads
  // a third less per FLOP) but wastes one of its SMs where an expert has an odd number of tiles, and rounds are counted
  // in whole tiles.  So the rounds of both are estimated, every expert ending in half a tile or pair on average.
  // Forward and backward of a layer, E 64 H 2048 F 1024, GEMM times on single SMs / pairs: 2048 rows per expert 2741 /
  // 2591 us, 1000 1449 / 1336, 500 788 / 752, 250 514 / 527.  E 8 H 4096 F 14336 at 512 rows: 918 / 843 where 28
  // rounds of tiles face 31 of pairs, 428 / 471 where 4 face 5.
  const double tiles = pt.n_slots / 128.0 + 0.5 * pt.E, pairs = pt.n_slots / 256.0 + 0.5 * pt.E;
  const int64_t cols = (N + (epilogue == cmoe::EPI_SWIGLU_FWD ? 127 : 255)) / (epilogue == cmoe::EPI_SWIGLU_FWD ? 128 : 256);
  // Near a tie it depends on the experts' loads, which the host does not know: with equal ones pairs win, where a few experts
  // have most rows single SMs, which compute fewer rows of padding, and more so in long runs at the power limit (these, seconds
  // of calls).  Pairs / single SMs in training, whose losses even the loads out: 800 tokens top-8, E 32 H 4096 F 2048 1781 /
  // 1810 us with unequal loads and 1656 / 1744 with equal ones, 1500 tokens 2435 / 2484 and 2407 / 2480, 512 tokens 1550 /
  // 1522 and 1500 / 1560, 1300 tokens E 64 H 2048 F 1024 935 / 938 and 915 / 955.  In inference: 7 rounds of pairs against 6
  // of tiles, 512 tokens 475 / 437 and 441 / 453, 1000 tokens 263 / 260 and 249 / 245, two decoder layers of that kind 868 /
  // 847; 8 against 7, 1300 tokens 288 / 282 and 267 / 297; 9 against 8, 800 tokens 554 / 545 and 473 / 527.
  if ((training ? 0.85 : 0.87) * std::ceil(pairs * cols / (g.num_sms / 2)) < std::ceil(tiles * cols / g.num_sms)) {
    g.pair_tile = plan + pt.pair_tile;
    g.num_pairs = plan + pt.num_pairs;
  }
  return g;
}

// The row plan of `idx32` [N, K] over all E experts; capacity > 0: slots kept per (expert, k)
Tensor build_plan(const Tensor& idx32, int64_t E, int64_t capacity, const OptTensor& overflow, cudaStream_t stream) {
  const PlanTables pt(idx32.numel(), E);
  const int K = static_cast<int>(idx32.size(1)), per_k = capacity > 0;
  Tensor plan_t = at::empty({pt.words}, idx32.options());
  Tensor scratch = at::empty(
      {static_cast<int64_t>(cmoe::moe_plan_scratch_words(pt.n_slots, static_cast<int>(E), K, per_k))}, idx32.options());
  int* plan = plan_t.data_ptr<int>();
  cmoe::MoePlanArgs a;
  a.topk_idx = idx32.data_ptr<int>();
  a.n_slots = pt.n_slots;
  a.K = K;
  a.num_experts = a.n_local = static_cast<int>(E);
  a.per_k_bins = per_k;
  a.capacity = static_cast<int>(capacity);
  a.cap_rows = pt.cap_rows;
  a.slot_row = plan;
  a.row_slot = plan + pt.row_slot;
  a.group_offsets = plan + pt.group_offsets;
  a.tile_group = plan + pt.tile_group;
  a.pair_tile = plan + pt.pair_tile;
  a.num_pairs = plan + pt.num_pairs;
  a.tile_rows = plan + pt.tile_rows;
  a.group_order = plan + pt.group_order;
  a.num_m_tiles = plan + pt.num_m_tiles;
  a.counts_kept = plan + pt.counts_kept;
  a.scratch = scratch.data_ptr<int>();
  a.overflow = status_ptr(overflow);
  check(cmoe::launch_moe_plan(a, stream), "moe_plan");
  return plan_t;
}
// ... as a call of its own, and its tables by name (views), for checks between the plan and the kernels that read it
Tensor moe_local_plan(const Tensor& idx32, int64_t E, int64_t capacity, const OptTensor& overflow) {
  TORCH_CHECK(idx32.is_cuda() && idx32.scalar_type() == at::kInt && idx32.dim() == 2 && idx32.is_contiguous(),
              "idx must be contiguous int32 [N, K]");
  const c10::cuda::CUDAGuard guard(idx32.device());
  return build_plan(idx32, E, capacity, overflow, at::cuda::getCurrentCUDAStream().stream());
}
std::map<std::string, Tensor> moe_local_tables(const Tensor& plan, int64_t n_slots, int64_t E) {
  const PlanTables pt(n_slots, E);
  TORCH_CHECK(plan.dim() == 1 && plan.numel() == pt.words, "the row plan belongs to another layer call");
  const int64_t tiles = pt.cap_rows / 128;
  const auto part = [&](int64_t at, int64_t n) { return plan.narrow(0, at, n); };
  return {{"slot_row", part(0, n_slots)},
          {"row_slot", part(pt.row_slot, pt.cap_rows)},
          {"group_offsets", part(pt.group_offsets, E + 1)},
          {"tile_group", part(pt.tile_group, tiles)},
          {"pair_tile", part(pt.pair_tile, tiles)},
          {"num_pairs", part(pt.num_pairs, 1)},
          {"tile_rows", part(pt.tile_rows, tiles)},
          {"group_order", part(pt.group_order, E)},
          {"num_m_tiles", part(pt.num_m_tiles, 1)},
          {"counts_kept", part(pt.counts_kept, E)}};
}

// the rows of `src` (tokens) and their places in expert order
cmoe::PlaceRowsArgs places(const Tensor& src, const Tensor& out, int64_t K, const PlanTables& pt, const int* plan,
                           bool zero_padding) {
  cmoe::PlaceRowsArgs a;
  a.src = src.data_ptr();
  a.n_tokens = src.size(0);
  a.ld_src = src.stride(0);
  a.slot_row = plan;
  a.K = static_cast<int>(K);
  a.H = static_cast<int>(src.size(1));
  a.out = out.data_ptr();
  a.ld_out = out.stride(0);
  a.zero_padding = zero_padding;
  a.group_offsets = plan + pt.group_offsets;
  a.counts_kept = plan + pt.counts_kept;
  a.n_local = static_cast<int>(pt.E);
  return a;
}

// (y, plan, xp, hact, gu, yp); the last four only with `keep` (what the backward reads)
Forward moe_local_forward(const Tensor& x, const Tensor& gate_w32, const Tensor& idx32, const Tensor& w13,
                          const Tensor& w2, int64_t capacity, bool keep, const OptTensor& status,
                          const OptTensor& overflow, const OptTensor& made_plan) {
  const c10::cuda::CUDAGuard guard(x.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
  const Shapes s = check_shapes(x, idx32, w13, w2);
  TORCH_CHECK(gate_w32.scalar_type() == at::kFloat && gate_w32.is_contiguous() && gate_w32.numel() == s.N * s.K,
              "gate weights must be contiguous fp32 [N, K]");
  const PlanTables pt(s.N * s.K, s.E);
  const auto bf = x.options();
  const Tensor plan_t = made_plan.has_value() ? *made_plan : build_plan(idx32, s.E, capacity, overflow, stream);
  TORCH_CHECK(plan_t.scalar_type() == at::kInt && plan_t.numel() == pt.words, "the row plan belongs to another layer call");
  int* plan = plan_t.data_ptr<int>();
  // Without a backward pass nobody reads the padding rows, so they are not filled, and where experts have few rows the
  // GEMMs load and store only the 32-row pieces that hold any: at 64 tokens, E 64 top-8 (8 rows per expert), H 2048,
  // F 1024 the padding was 33 MB to fill, 400 MB to load from L2 and 50 MB to store, next to 805 MB of weights.  From 64
  // rows per expert on, most pieces are live and whole tiles take fewer loads.
  const bool short_tiles = !keep && pt.n_slots <= 64 * s.E;
  Tensor xp = at::empty({pt.cap_rows, s.H}, bf);
  check(cmoe::launch_place_rows(places(x, xp, s.K, pt, plan, keep), stream), "place_rows");
  Tensor hact = at::empty({pt.cap_rows, s.F}, bf);
  OptTensor gu;
  {
    cmoe::GemmArgs g = grouped_rows(xp, w13, 2 * s.F, false, hact, s.F, s.H, pt, plan, status_ptr(status), cmoe::EPI_SWIGLU_FWD,
                                     keep, short_tiles);
    g.split_n = static_cast<int>(s.F);
    if (keep) {
      gu = at::empty({pt.cap_rows, 2 * s.F}, bf);
      g.aux_out = gu->data_ptr();
      g.ld_aux_out = 2 * s.F;
    }
    cmoe::launch_gemm_any(g, stream);
  }
  Tensor yp = at::empty({pt.cap_rows, s.H}, bf);
  cmoe::launch_gemm_any(grouped_rows(hact, w2, s.H, false, yp, s.H, s.F, pt, plan, status_ptr(status),
                                      cmoe::EPI_STORE, keep, short_tiles),
                         stream);
  Tensor y = at::empty({s.N, s.H}, bf);
  check(cmoe::launch_combine_rows(yp.data_ptr(), plan, gate_w32.data_ptr<float>(), y.data_ptr(), s.N,
                                  static_cast<int>(s.K), static_cast<int>(s.H), s.H, s.H, stream),
        "combine_rows");
  if (!keep) return {y, plan_t, std::nullopt, std::nullopt, std::nullopt, std::nullopt};
  return {y, plan_t, xp, hact, gu, yp};
}

// dW[e] = a[rows of e]^T b[rows of e]: added into the fp32 `main` buffer when there is one (returns nothing), else
// rounded once into a new tensor of the weight's type
OptTensor expert_wgrad(const Tensor& a, const Tensor& b, const Tensor& weight, const OptTensor& main, const PlanTables& pt,
                       const int* plan, int* status, cudaStream_t stream) {
  cmoe::GemmArgs g;
  g.A = a.data_ptr();
  g.a_rows = a.size(0);
  g.a_cols = a.size(1);
  g.a_ld = a.stride(0);
  g.a_mn = 1;
  g.B = b.data_ptr();
  g.b_rows = b.size(0);
  g.b_cols = b.size(1);
  g.b_ld = b.stride(0);
  g.b_mn = 1;
  g.mode = cmoe::GEMM_GROUPED_K;
  g.M = static_cast<int>(a.size(1));
  g.N = static_cast<int>(b.size(1));
  g.groups = static_cast<int>(pt.E);
  g.group_offsets = plan + pt.group_offsets;
  g.d_group_stride = a.size(1) * b.size(1);
  g.ldd = b.size(1);
  g.status = status;
  g.num_sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  // Longest experts first, so that unequal ones fill the pairs of SMs evenly: E 64 H 2048 F 1024, 2048 rows per expert
  // (the busiest three times that) 1479 -> 1288 us for both weights, E 16 H 704 F 320, 625 rows 41 -> 34.  Not over
  // many rounds of tiles of few rows, which are bound by the stores of their results: in the experts' own order these
  // overlap the arithmetic of longer neighbours (500 rows per expert 424 us in their own order, 456 sorted).
  const int64_t rounds = ((g.M + 255) / 256) * ((g.N + 255) / 256) * pt.E / (g.num_sms / 2);
  if (rounds <= 16 || (rounds <= 64 && pt.n_slots >= 1024 * pt.E)) g.group_order = plan + pt.group_order;
  OptTensor out;
  if (main.has_value()) {
    TORCH_CHECK(main->scalar_type() == at::kFloat && main->is_contiguous() && main->numel() == weight.numel(),
                "main_grad must be a contiguous fp32 tensor of the weight's shape");
    g.D = main->data_ptr();
    g.d_fp32 = g.accumulate = 1;
  } else {
    out = at::empty(weight.sizes(), weight.options());
    g.D = out->data_ptr();
  }
  cmoe::launch_gemm_any(g, stream);
  return out;
}

// (dx, d_gate, dw13, dw2).  Everything but dy is a saved tensor, which a hook may hand back in another layout: brought into
// the kernels' one, or refused.
Backward moe_local_backward(const Tensor& dy, const Tensor& saved_plan, const Tensor& saved_xp, const Tensor& saved_hact,
                            const Tensor& saved_gu, const Tensor& saved_yp, const Tensor& saved_gate, const Tensor& saved_w13,
                            const Tensor& saved_w2, bool need_dx, bool need_gate, const OptTensor& main13,
                            const OptTensor& main2, const OptTensor& status) {
  const c10::cuda::CUDAGuard guard(dy.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
  const Tensor plan_t = cmoe::contiguous_aligned(saved_plan), xp = cmoe::contiguous_aligned(saved_xp),
               hact = cmoe::contiguous_aligned(saved_hact), gu = cmoe::contiguous_aligned(saved_gu),
               yp = cmoe::contiguous_aligned(saved_yp), gate_w32 = cmoe::contiguous_aligned(saved_gate),
               w13 = cmoe::contiguous_aligned(saved_w13), w2 = cmoe::contiguous_aligned(saved_w2);
  TORCH_CHECK(gate_w32.dim() == 2 && xp.dim() == 2 && hact.dim() == 2 && w13.dim() == 3, "bad saved tensors");
  const int64_t N = gate_w32.size(0), K = gate_w32.size(1), H = xp.size(1), E = w13.size(0), F = hact.size(1);
  TORCH_CHECK(dy.scalar_type() == at::kBFloat16 && dy.is_contiguous() && dy.size(0) == N && dy.size(1) == H, "bad dy");
  check_rows(dy, "dy");
  check_rows(xp, "saved rows");
  check_rows(yp, "saved expert rows");
  const PlanTables pt(N * K, E);
  const auto is = [&](const Tensor& t, at::ScalarType type, at::IntArrayRef sizes) {
    return t.device() == dy.device() && t.scalar_type() == type && t.sizes() == sizes;
  };
  TORCH_CHECK(is(plan_t, at::kInt, {pt.words}) && is(xp, at::kBFloat16, {pt.cap_rows, H}),
              "the row plan belongs to another layer call");
  TORCH_CHECK(is(hact, at::kBFloat16, {pt.cap_rows, F}) && is(gu, at::kBFloat16, {pt.cap_rows, 2 * F}) &&
                  is(yp, at::kBFloat16, {pt.cap_rows, H}) && is(gate_w32, at::kFloat, {N, K}) &&
                  is(w13, at::kBFloat16, {E, 2 * F, H}) && is(w2, at::kBFloat16, {E, H, F}),
              "the saved tensors of the expert layer are not what its forward left");
  int* plan = plan_t.data_ptr<int>();
  int* st = status_ptr(status);
  Backward out;
  Tensor dyp = at::empty({pt.cap_rows, H}, dy.options()), d_gate;
  if (need_gate) d_gate = at::empty({N, K}, gate_w32.options());
  float* dw = need_gate ? d_gate.data_ptr<float>() : nullptr;
  if (cmoe::combine_grad_supported(static_cast<int>(H))) {
    check(cmoe::launch_combine_grad(places(dy, dyp, K, pt, plan, true), gate_w32.data_ptr<float>(), yp.data_ptr(), H, dw, stream),
          "combine_grad");
  } else {  // rows that do not fit a warp's registers
    if (need_gate)
      check(cmoe::launch_combine_bwd_w(yp.data_ptr(), plan, dy.data_ptr(), dw, N, static_cast<int>(K), static_cast<int>(H), H,
                                       H, stream),
            "combine_bwd_w");
    check(cmoe::launch_gather_rows(dy.data_ptr(), plan + pt.row_slot, static_cast<int>(K), gate_w32.data_ptr<float>(),
                                   dyp.data_ptr(), pt.cap_rows, plan + pt.num_m_tiles, static_cast<int>(H), H, H, stream),
          "gather_rows");
  }
  if (need_gate) std::get<1>(out) = d_gate;
  Tensor dgu = at::empty({pt.cap_rows, 2 * F}, dy.options());
  {
    cmoe::GemmArgs g = grouped_rows(dyp, w2, H, true, dgu, F, H, pt, plan, st, cmoe::EPI_SWIGLU_BWD);
    g.aux_in = gu.data_ptr();
    g.ld_aux_in = gu.stride(0);
    cmoe::launch_gemm_any(g, stream);
  }
  if (need_dx) {
    Tensor dxp = at::empty({pt.cap_rows, H}, dy.options());
    cmoe::launch_gemm_any(grouped_rows(dgu, w13, 2 * F, true, dxp, H, 2 * F, pt, plan, st), stream);
    Tensor dx = at::empty({N, H}, dy.options());
    check(cmoe::launch_combine_rows(dxp.data_ptr(), plan, nullptr, dx.data_ptr(), N, static_cast<int>(K),
                                    static_cast<int>(H), H, H, stream),
          "combine_rows");
    std::get<0>(out) = dx;
  }
  std::get<3>(out) = expert_wgrad(dyp, hact, w2, main2, pt, plan, st, stream);
  std::get<2>(out) = expert_wgrad(dgu, xp, w13, main13, pt, plan, st, stream);
  return out;
}

}  // namespace

namespace cmoe {
MoeForward moe_local_forward(const Tensor& x, const Tensor& gate_w32, const Tensor& idx32, const Tensor& w13,
                             const Tensor& w2, int64_t capacity, bool keep, const OptTensor& status,
                             const OptTensor& overflow, const OptTensor& made_plan) {
  return ::moe_local_forward(x, gate_w32, idx32, w13, w2, capacity, keep, status, overflow, made_plan);
}
MoeBackward moe_local_backward(const Tensor& dy, const Tensor& plan, const Tensor& xp, const Tensor& hact, const Tensor& gu,
                               const Tensor& yp, const Tensor& gate_w32, const Tensor& w13, const Tensor& w2,
                               bool need_dx, bool need_gate, const OptTensor& main13, const OptTensor& main2,
                               const OptTensor& status) {
  return ::moe_local_backward(dy, plan, xp, hact, gu, yp, gate_w32, w13, w2, need_dx, need_gate, main13, main2, status);
}
}  // namespace cmoe

void register_moe(pybind11::module_& m) {
  m.def("moe_local_plan", &moe_local_plan);
  m.def("moe_local_tables", &moe_local_tables);
  m.def("moe_local_forward", &moe_local_forward);
  m.def("moe_local_backward", &moe_local_backward);
}
