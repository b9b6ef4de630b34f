// Fused top-k router for sm_100a.
//
// Forward, one launch: gate GEMM (tokens [N,H] x gate_w [H,E]) on tcgen05 with the fp32 logits in
// tensor memory, then per token row out of shared memory: top-k with lowest-index tie break, fp32 softmax
// statistics, renormalised gate weights, per-expert counts, per-expert probability sums (load-balance loss),
// z-loss, and a last-CTA finalisation that turns those sums into the loss values.  The tokens are read from HBM
// exactly once.
//
// What bounds it: with many tokens the read of the tokens, with few tokens (or many experts) what one SM can pull
// in, and in both cases the epilogue that no other work hides.  Hence
//   * a tile has 128 rows only where the tokens fill the GPU with such tiles; fewer tokens get tiles of 64, 32 or 16
//     rows (the MMA still computes 128, the rows that were not loaded are never read back), so that more SMs share the
//     epilogue;
//   * 128 and more experts on few tiles are split over a cluster of CTAs, each with its share of the experts and of the
//     gate weights, which every tile reads whole; the logits meet through distributed shared memory and every CTA
//     finishes its share of the rows.  (Splitting H instead would add the logits up in another order, and with it
//     decide near-ties between experts differently for different token counts.);
//   * every k-block costs its issue: on few tokens the loop over H is as long as single threads need to wait, load and
//     issue.  The gate weights have a loading warp of their own, two k-blocks share a barrier, and the MMA loop only
//     advances its descriptors (590 -> 310 cycles per k-block of 64);
//   * the epilogue runs on 16 warps with four lanes per row over logits in shared memory.  A thread per row straight
//     out of tensor memory took longer than the GEMM: 54 us of 88 at 8190 tokens, E 256, top-8.
// Launch to end with a cold L2, first form (128-row tiles, a thread per row) and now: 8190 tokens H 4096 E 256 top-8
// 94 -> 47 us, 64 x 2048 E 64 top-8 33 -> 25, 1000 x 2048 E 64 top-8 35 -> 25, 16384 x 2048 E 64 top-8 41 -> 35,
// 16384 x 4096 E 64 top-2 51 -> 47 (134 MB of tokens: 21 us at the copy rate).
//
// Gate weights are exp(v - lse) over their sum, with lse and that sum added in a fixed order (see the epilogue).
//
// Backward: the analytic gradient of the gate weights, load-balance loss and z-loss with respect
// to the logits (eight lanes per token); the two contractions with it (grad_tokens, grad_gate_w) run
// on the tcgen05 GEMMs (host_ops.cpp: dense_nt, dense_wgrad).
//
// Counterpart in the reference: the Triton kernels _router_fwd_kernel / _router_bwd_kernel plus the
// bincount, the second logits GEMM for the z-loss and the two cuBLAS GEMMs of the backward
// (pkg/kernels/moe_router.py:102-251, 545-546, 690-734).
#include "router.cuh"

#include <climits>

#include "common.cuh"
#include "launch.h"
#include "tensor_maps.h"

namespace cmoe {

namespace {

constexpr int RT_BM = 128;
constexpr int RT_BK = 64;
constexpr int RT_CHUNK_BYTES = 64 * RT_BK * 2;  // 8 KiB: 64 experts x 64 k
constexpr int RT_EPI = 512;                     // epilogue threads (warps 2..17)
constexpr int RT_W_WARP = 2 + RT_EPI / 32;      // the last warp: loads of the gate weights
constexpr int RT_THREADS = 96 + RT_EPI;
constexpr int RT_SUB = 2;  // k-blocks of a stage: one wait and one commit for eight MMAs
constexpr int RT_MAX_STAGES = 12;
constexpr int RT_SMEM_BUDGET = 200 * 1024;

struct RouterParams {
  long long n_tokens;
  int H, E, K;
  int rows;      // rows of a tile that are loaded: 128, 64, 32 or 16
  int split;     // CTAs per row tile (the cluster size): each takes its share of the experts
  int n_chunks;  // 64-expert chunks of the gate weights that one CTA loads
  int stages;
  int umma_n;  // experts of one CTA, rounded up to 16
  int tmem_cols;
  float* logits;
  int* topk_idx;
  float* topk_w;
  long long* topk_idx64;
  __nv_bfloat16* topk_w16;
  float* lse;
  int* counts;
  long long* counts64;
  float* mean_prob;
  float* stats;  // nullptr: no statistics are gathered
  uint32_t* workspace;
  int* status;
  unsigned long long timeout_ns;
};

// groups of eight experts per lane, the kernel's template argument
__host__ __device__ constexpr int rt_groups(int E) { return E <= 32 ? 1 : E <= 64 ? 2 : E <= 128 ? 4 : 8; }
// row stride (floats) of the logits tile in shared memory: room for every expert that the lanes of that variant look at
// (the columns past E are masked out, but no other row's), and 4 more than a multiple of 32 banks, so that both the
// 16-byte stores of 32 neighbouring rows and the reads of 8 rows x 4 lanes touch every bank once
__host__ __device__ constexpr int rt_row_stride(int groups) { return 32 * groups + 4; }
// per-CTA tables behind the pipeline stages (bytes); the barriers come first
constexpr int RT_TABLES = 1024 /* barriers, slots */ + RT_BM * 4 /* 1/sum */ + RT_BM * 4 /* lse^2 */ + RT_EPI * 4 /* column partials */ +
                          kRouterMaxExperts * 4 /* counts */ + 2 * kRouterMaxTopK * RT_BM * 4 /* picks */;

// order-preserving map of a logit to an integer: +0 and -0 agree, NaN takes a place at the end of the order (so every
// pick is a valid expert whatever the input), and nothing maps to INT_MIN, which stands for "taken"
__device__ __forceinline__ int logit_key(float v) {
  const int b = __float_as_int(v + 0.f);
  return max(b ^ ((b >> 31) & 0x7fffffff), INT_MIN + 1);
}
__device__ __forceinline__ float key_logit(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ uint32_t rt_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void rt_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void rt_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t smem_addr, uint32_t rank) {
  float4 v;
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// NG: groups of eight experts per lane (a row's four lanes take the experts 4 j + lane): E <= 32 NG
template <int NG>
__global__ void __launch_bounds__(RT_THREADS, 1)
router_fwd_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                  const RouterParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int b_bytes = p.n_chunks * RT_CHUNK_BYTES;
  const int a_bytes = p.rows * RT_BK * 2;
  const int stage_bytes = RT_SUB * (a_bytes + b_bytes);
  constexpr int SE = rt_row_stride(NG);
  static_assert(SE >= 32 * NG, "a row has a cell for every expert its lanes look at");
  const int front = max(p.stages * stage_bytes, p.rows * SE * 4);
  float* s_logit = reinterpret_cast<float*>(smem);  // [rows][SE], over the drained pipeline stages
  // behind all of A: what an MMA reads past a short tile's rows is ours
  uint8_t* sB = smem + p.stages * RT_SUB * a_bytes;
  uint8_t* tail = smem + front;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(tail);   // [RT_MAX_STAGES]
  uint64_t* empty_bar = full_bar + RT_MAX_STAGES;           // [RT_MAX_STAGES]
  uint64_t* tfull_bar = empty_bar + RT_MAX_STAGES;          // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_last = const_cast<int*>(abort_flag) + 1;
  float* s_inv = reinterpret_cast<float*>(tail + 1024);  // [128] 1 / sum of exponentials (0: no such token)
  float* s_z = s_inv + RT_BM;                           // [128] lse^2
  float* s_part = s_z + RT_BM;                          // [512] column sums of row ranges
  int* s_cnt = reinterpret_cast<int*>(s_part + RT_EPI);        // [256]
  int* s_topi = s_cnt + kRouterMaxExperts;                     // [kRouterMaxTopK][128] chosen experts
  float* s_topv = reinterpret_cast<float*>(s_topi + kRouterMaxTopK * RT_BM);  // ... their logits, then gate weights

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int split = p.split;
  const int rank = split > 1 ? static_cast<int>(rt_cluster_rank()) : 0;
  const long long row0 = static_cast<long long>(blockIdx.x / split) * p.rows;
  const int k_blocks = (p.H + RT_BK - 1) / RT_BK;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *s_last = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 2);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tfull_bar, 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_wait();
  chain_trigger();

  WaitCtx wc;
  wc.abort_flag = abort_flag;
  wc.status = p.status;
  wc.timeout_ns = p.timeout_ns;

  const int et = static_cast<int>(threadIdx.x) - 64;  // epilogue thread
  const int E = p.E;
  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < k_blocks; kb += RT_SUB) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u, wc, ST_TIMEOUT_SMEM_EMPTY)) break;
        const int sub = min(RT_SUB, k_blocks - kb);
        mbar_arrive_expect_tx(&full_bar[stage], sub * a_bytes);
        for (int s = 0; s < sub; ++s)
          tma_load_2d(smem + (stage * RT_SUB + s) * a_bytes, &tmX, &full_bar[stage], (kb + s) * RT_BK,
                      static_cast<int>(row0));
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == RT_W_WARP) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < k_blocks; kb += RT_SUB) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u, wc, ST_TIMEOUT_SMEM_EMPTY)) break;
        const int sub = min(RT_SUB, k_blocks - kb);
        mbar_arrive_expect_tx(&full_bar[stage], sub * b_bytes);
        for (int s = 0; s < sub; ++s) {
          uint8_t* b_dst = sB + (stage * RT_SUB + s) * b_bytes;
          for (int j = 0; j < p.n_chunks; ++j)
            tma_load_2d(b_dst + j * RT_CHUNK_BYTES, &tmW, &full_bar[stage], 64 * (rank * p.n_chunks + j),
                        (kb + s) * RT_BK);
        }
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
      const uint64_t b_desc0 = make_smem_desc_sw128(smem_u32(sB), RT_CHUNK_BYTES, 1024);
      const uint32_t idesc = make_idesc_bf16(RT_BM, p.umma_n, 0, 1);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < k_blocks; kb += RT_SUB) {
        if (!mbar_wait(&full_bar[stage], phase, wc, ST_TIMEOUT_SMEM_FULL)) break;
        tc_fence_after();
        const int sub = min(RT_SUB, k_blocks - kb);
        for (int q = 0; q < sub; ++q) {
          const uint64_t ad = a_desc0 + static_cast<uint32_t>((stage * RT_SUB + q) * (a_bytes >> 4));
          const uint64_t bd = b_desc0 + static_cast<uint32_t>((stage * RT_SUB + q) * (b_bytes >> 4));
#pragma unroll
          for (int k = 0; k < RT_BK / 16; ++k)
            umma_bf16_ss(tmem_base, ad + k * (32 >> 4), bd + k * (2048 >> 4), idesc, (kb | q | k) != 0 ? 1u : 0u);
        }
        umma_commit(&empty_bar[stage]);
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      umma_commit(tfull_bar);
    }
    __syncwarp();
  } else {
    for (int e = et; e < kRouterMaxExperts; e += RT_EPI) s_cnt[e] = 0;
    const bool ok = mbar_wait(tfull_bar, 0, wc, ST_TIMEOUT_TMEM_FULL);
    tc_fence_after();
    if (ok) {
      // logits: tensor memory -> shared memory, every warp its own quadrant of lanes and every fourth 16 columns
      const int quad = warp & 3;
      const int e_cta = E / split;  // this CTA's experts
      float* dst = s_logit + (quad * 32 + lane) * SE + rank * e_cta;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
      const int c_end = quad * 32 < p.rows ? e_cta : 0;
#pragma unroll 1
      for (int c = (et >> 7) * 16; c < c_end; c += 64) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_row + c, r);
        tmem_ld_wait();
        if (quad * 32 + lane < p.rows) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)  // the row stride has room for all 16 columns
            *reinterpret_cast<float4*>(dst + c + j) = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]),
                                                                  __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
        }
        __syncwarp();
      }
    }
    __syncwarp();
  }
  if (split > 1) {  // every CTA's logits are in its shared memory
    rt_cluster_arrive();
    rt_cluster_wait();
  }
  if (warp >= 2 && warp != RT_W_WARP) {
    const int R = p.rows / split;  // this CTA finishes the rows [r_lo, r_lo + R) of the tile
    const int r_lo = rank * R;
    if (split == 1) epi_sync();
    // bring in the logits that the other CTAs of the cluster computed; the logits go out to global memory
    if (split > 1 || p.logits != nullptr) {
      constexpr int C4 = 8 * NG;  // threads of a row, 16 bytes each
      const int c = (et & (C4 - 1)) * 4;
      if (c < E) {
        const int owner = split > 1 ? c / (E / split) : rank;
#pragma unroll 4
        for (int r = et / C4; r < R; r += RT_EPI / C4) {
          float* cell = s_logit + (r_lo + r) * SE + c;
          float4 v;
          if (owner != rank) {
            v = ld_cluster_f4(smem_u32(cell), owner);
            *reinterpret_cast<float4*>(cell) = v;
          } else {
            v = *reinterpret_cast<const float4*>(cell);
          }
          const long long row = row0 + r_lo + r;
          if (p.logits != nullptr && row < p.n_tokens) *reinterpret_cast<float4*>(p.logits + row * E + c) = v;
        }
      }
      if (split > 1) epi_sync();
    }
  }
  if (split > 1) rt_cluster_arrive();  // done with the other CTAs' shared memory; waited for before the exit
  if (warp >= 2 && warp != RT_W_WARP) {
    const int R = p.rows / split;
    const int r_lo = rank * R;
    const int t = et >> 2, l = et & 3;  // row of this CTA's share, lane of the row
    const int n = E / 4;                // experts per lane (E is a multiple of 8)
    const long long row = row0 + r_lo + t;
    const bool row_ok = row < p.n_tokens;
    if (t < R) {  // whole warps: R is a multiple of 8
      float* mine = s_logit + (r_lo + t) * SE + l;
      // best of every group of eight of this lane's experts
      int gk[NG], gj[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        gk[g] = INT_MIN;
        gj[g] = g * 8;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int j = g * 8 + q;
          const float v = mine[4 * j];  // columns past E lie inside the row stride, and are masked out
          const int k = j < n ? logit_key(v) : INT_MIN;
          if (k > gk[g]) {
            gk[g] = k;
            gj[g] = j;
          }
        }
      }
      // top-k: best group, best of the four lanes, then the winning lane looks through its one group again.  The loop
      // over k stays rolled: this code runs once per CTA, so every instruction is a cold fetch.
      unsigned long long taken = 0ull;
#pragma unroll 1
      for (int kk = 0; kk < p.K; ++kk) {
        int bk = gk[0], bj = gj[0];
#pragma unroll
        for (int g = 1; g < NG; ++g)
          if (gk[g] > bk) {
            bk = gk[g];
            bj = gj[g];
          }
        int e = 4 * bj + l;
#pragma unroll
        for (int off = 1; off <= 2; off <<= 1) {
          const int ok = __shfl_xor_sync(0xffffffffu, bk, off), oe = __shfl_xor_sync(0xffffffffu, e, off);
          if (ok > bk || (ok == bk && oe < e)) {
            bk = ok;
            e = oe;
          }
        }
        if (l == 0) {
          s_topi[kk * RT_BM + t] = e;
          s_topv[kk * RT_BM + t] = key_logit(bk);
        }
        if (l == (e & 3)) {
          const int wj = e >> 2, wg = wj >> 3;
          taken |= 1ull << wj;
          const uint32_t tk = static_cast<uint32_t>(taken >> (wg * 8));
          const float* grp = mine + 32 * wg;
          float v8[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) v8[q] = grp[4 * q];
          int nk = INT_MIN, nj = wg * 8;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int k = (wg * 8 + q < n && ((tk >> q) & 1u) == 0u) ? logit_key(v8[q]) : INT_MIN;
            if (k > nk) {
              nk = k;
              nj = wg * 8 + q;
            }
          }
#pragma unroll
          for (int g = 0; g < NG; ++g)
            if (g == wg) {
              gk[g] = nk;
              gj[g] = nj;
            }
        }
        __syncwarp();
      }
      // Softmax statistics; the exponentials replace the logits, and the first pick is the row maximum.  The log-sum-exp
      // adds them in the order of the experts and the gate weights exp(v - lse) are added in the order of the picks,
      // whatever the tile, the cluster or the lanes: a last bit of a gate weight moves roundings in all that follows, and
      // with top-1 routing, where the weight is 1, the rounding of lse is all that its gradient consists of.  All four
      // lanes add the same E numbers (16-byte reads that they share).  Where only the decision is wanted this costs 1.5 us
      // of 28 (16384 x 4096, E 64, top-2); with statistics, which need the exponentials anyway, at most one.
      const float mx = s_topv[t];
#pragma unroll 8
      for (int j = 0; j < n; ++j) mine[4 * j] = expf(mine[4 * j] - mx);
      __syncwarp();
      const float4* ex = reinterpret_cast<const float4*>(mine - l);
      float se = 0.f;
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        const float4 v = ex[j];
        se += v.x;
        se += v.y;
        se += v.z;
        se += v.w;
      }
      const float lse = mx + logf(se);
      // gate weights: lane l takes the picks l and l + 4
      const float w0 = l < p.K ? expf(s_topv[l * RT_BM + t] - lse) : 0.f;
      const float w1 = l + 4 < p.K ? expf(s_topv[(l + 4) * RT_BM + t] - lse) : 0.f;
      if (l < p.K) s_topv[l * RT_BM + t] = w0;
      if (l + 4 < p.K) s_topv[(l + 4) * RT_BM + t] = w1;
      __syncwarp();
      float psum = 0.f;
      for (int kk = 0; kk < p.K; ++kk) psum += s_topv[kk * RT_BM + t];
      const float inv_psum = 1.f / psum;
      __syncwarp();
      if (l < p.K) s_topv[l * RT_BM + t] = w0 * inv_psum;
      if (l + 4 < p.K) s_topv[(l + 4) * RT_BM + t] = w1 * inv_psum;
      if (l == 0) {
        if (row_ok && p.lse != nullptr) p.lse[row] = lse;
        s_inv[t] = row_ok ? 1.f / se : 0.f;
        s_z[t] = row_ok ? lse * lse : 0.f;
      }
    }
    epi_sync();
    // the picks, whole rows of K at a time
    const int live = static_cast<int>(min(static_cast<long long>(R), p.n_tokens - (row0 + r_lo)));
    for (int i = et; i < live * p.K; i += RT_EPI) {
      const int r = i / p.K, kk = i - r * p.K;
      const long long o = (row0 + r_lo) * p.K + i;
      const int e = s_topi[kk * RT_BM + r];
      const float w = s_topv[kk * RT_BM + r];
      atomicAdd(&s_cnt[e], 1);
      if (p.topk_idx != nullptr) p.topk_idx[o] = e;
      if (p.topk_idx64 != nullptr) p.topk_idx64[o] = e;
      if (p.topk_w != nullptr) p.topk_w[o] = w;
      if (p.topk_w16 != nullptr) p.topk_w16[o] = __float2bfloat16(w);
    }
    if (p.stats != nullptr) {
      // probability sums: thread = (expert, range of rows), then the ranges of an expert in order
      const int cols = NG == 1 ? 32 : (NG == 2 ? 64 : (NG == 4 ? 128 : 256));
      const int parts = RT_EPI / cols, per = (R + parts - 1) / parts;
      const int e = et & (cols - 1), part = et / cols;
      float sum = 0.f;
      if (e < E) {
        const int r1 = min(R, (part + 1) * per);
#pragma unroll 8
        for (int r = part * per; r < r1; ++r) sum += s_logit[(r_lo + r) * SE + e] * s_inv[r];
      }
      s_part[part * cols + e] = sum;
      epi_sync();
      // flush this share's sums as 64-bit fixed point (integer adds commute: the result does not depend on the order
      // of the CTAs); the last CTA to finish turns them into the loss values
      unsigned long long* ws_prob = reinterpret_cast<unsigned long long*>(p.workspace);
      unsigned long long* ws_z = ws_prob + E;
      int* ws_cnt = reinterpret_cast<int*>(ws_z + 1);
      unsigned int* ws_done = reinterpret_cast<unsigned int*>(ws_cnt + E);
      if (et < E) {
        float pr = 0.f;
        for (int q = 0; q < parts; ++q) pr += s_part[q * cols + et];
        const unsigned long long fx = __float2ull_rn(pr * kRouterProbScale);
        if (fx != 0ull) atomicAdd(&ws_prob[et], fx);
        if (s_cnt[et] != 0) atomicAdd(&ws_cnt[et], s_cnt[et]);
      } else if (et >= RT_EPI - 32) {  // E <= 256: this warp has no expert
        float z = 0.f;
        for (int r = lane; r < R; r += 32) z += s_z[r];
        z = warp_sum(z);
        if (lane == 0) atomicAdd(ws_z, __float2ull_rn(z * kRouterZScale));
      }
      __threadfence();
      epi_sync();
      if (et == 0) {
        const unsigned int ticket = atomicAdd(ws_done, 1u);
        *s_last = (ticket == gridDim.x - 1) ? 1 : 0;
      }
      epi_sync();
      if (*s_last) {
        __threadfence();
        const float n_tok = static_cast<float>(p.n_tokens);
        float aux = 0.f, mxc = 0.f, sumc = 0.f;
        if (et < E) {
          const float pr = static_cast<float>(static_cast<double>(__ldcg(&ws_prob[et])) / kRouterProbScale);
          const int cn = __ldcg(&ws_cnt[et]);
          if (p.counts != nullptr) p.counts[et] = cn;
          if (p.counts64 != nullptr) p.counts64[et] = cn;
          if (p.mean_prob != nullptr) p.mean_prob[et] = pr / n_tok;
          aux = (static_cast<float>(cn) / (n_tok * p.K)) * (pr / n_tok);
          mxc = static_cast<float>(cn);
          sumc = static_cast<float>(cn);
          ws_prob[et] = 0ull;
          ws_cnt[et] = 0;
        }
        aux = warp_sum(aux);
        mxc = warp_max(mxc);
        sumc = warp_sum(sumc);
        if (lane == 0) {
          const int w = et >> 5;
          s_part[w] = aux;
          s_part[16 + w] = mxc;
          s_part[32 + w] = sumc;
        }
        epi_sync();
        if (et == 0) {
          const int warps = (E + 31) / 32;
          for (int w = 1; w < warps; ++w) {
            aux += s_part[w];
            mxc = fmaxf(mxc, s_part[16 + w]);
            sumc += s_part[32 + w];
          }
          p.stats[0] = aux * E;
          p.stats[1] = static_cast<float>(static_cast<double>(__ldcg(ws_z)) / kRouterZScale) / n_tok;
          p.stats[2] = sumc > 0.f ? mxc / (sumc / E) : 1.f;
          p.stats[3] = sumc;
          *ws_z = 0ull;
          *ws_done = 0u;
        }
      }
    }
  }
  if (split > 1) rt_cluster_wait();  // nobody still reads this CTA's shared memory

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) {
      for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

// d(loss)/d(logits), eight lanes per token (four tokens per warp), logits in 16-byte pieces.  With p_i the softmax,
// g_i = d(loss)/d(p_i) = a_i + [i picked as k] d_k, the result is p_i (g_i - sum_j g_j p_j) + z-loss term; lane k
// holds pick k (K <= 8), so the sum over j splits into the dense part and the K picks, every lane writes its own
// dense values, and the lane of a pick then overwrites that one value.  A warp per token that compared every expert
// with every pick was bound by its instructions: 26.6 us at 16384 tokens, E 64, top-8 (6 MB).
__global__ void __launch_bounds__(256) router_bwd_kernel(const RouterBwdArgs a) {
  chain_wait();
  chain_trigger();
  const long long row_raw = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) >> 3;
  const int l = threadIdx.x & 7;
  const bool live = row_raw < a.n_tokens;
  const long long row = live ? row_raw : a.n_tokens - 1;  // idle lanes follow along for the shuffles
  const int E = a.E, K = a.K;
  const float* lg = a.logits + row * E;
  const float lse = a.lse[row];
  const float ga = a.grad_aux ? *a.grad_aux : 0.f;
  const float gz = a.grad_z ? *a.grad_z : 0.f;
  const float n_tok = static_cast<float>(a.n_tokens);
  const float aux_c = ga * E / (n_tok * n_tok * K);  // d(aux)/dp[t,i] = ga * E * (counts_i / (N K)) / N

  // lane l: pick l
  int pick = 0;
  float pk = 0.f, gw = 0.f;
  if (l < K) {
    pick = a.topk_idx[row * K + l];
    gw = a.grad_w ? a.grad_w[row * K + l] : 0.f;
    pk = expf(lg[pick] - lse);
  }
  float S = pk, gwv = gw * pk;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    S += __shfl_xor_sync(0xffffffffu, S, o);
    gwv += __shfl_xor_sync(0xffffffffu, gwv, o);
  }
  const float invS = 1.f / S;
  const float dk = l < K ? gw * invS - gwv * invS * invS : 0.f;

  float4 p[kRouterMaxExperts / 32];  // this lane's probabilities
  float dot = dk * pk;
#pragma unroll
  for (int q = 0; q < kRouterMaxExperts / 32; ++q) {
    const int e = (q * 8 + l) * 4;
    if (e < E) {
      const float4 v = *reinterpret_cast<const float4*>(lg + e);
      p[q] = make_float4(expf(v.x - lse), expf(v.y - lse), expf(v.z - lse), expf(v.w - lse));
      if (aux_c != 0.f) {
        const int4 c = *reinterpret_cast<const int4*>(a.counts + e);
        dot += aux_c * (p[q].x * c.x + p[q].y * c.y + p[q].z * c.z + p[q].w * c.w);
      }
    }
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  const float base = gz * 2.f * lse / n_tok - dot;
  __nv_bfloat16* out16 = reinterpret_cast<__nv_bfloat16*>(a.grad_logits_bf16);
#pragma unroll
  for (int q = 0; q < kRouterMaxExperts / 32; ++q) {
    const int e = (q * 8 + l) * 4;
    if (e < E && live) {
      float4 g = make_float4(base, base, base, base);
      if (aux_c != 0.f) {
        const int4 c = *reinterpret_cast<const int4*>(a.counts + e);
        g.x += aux_c * c.x; g.y += aux_c * c.y; g.z += aux_c * c.z; g.w += aux_c * c.w;
      }
      g.x *= p[q].x; g.y *= p[q].y; g.z *= p[q].z; g.w *= p[q].w;
      if (a.grad_logits_f32) *reinterpret_cast<float4*>(a.grad_logits_f32 + row * E + e) = g;
      if (out16) *reinterpret_cast<uint2*>(out16 + row * E + e) = make_uint2(pack_bf16x2(g.x, g.y), pack_bf16x2(g.z, g.w));
    }
  }
  __syncwarp();  // the dense values are written: now the picks
  if (l < K && live) {
    const float g = pk * (base + (aux_c != 0.f ? aux_c * a.counts[pick] : 0.f) + dk);
    if (a.grad_logits_f32) a.grad_logits_f32[row * E + pick] = g;
    if (out16) out16[row * E + pick] = __float2bfloat16(g);
  }
}

}  // namespace

template <int NG>
static cudaError_t launch_router_variant(const CUtensorMap& tmX, const CUtensorMap& tmW, const RouterParams& p,
                                         unsigned tiles, int smem, cudaStream_t stream) {
  static const cudaError_t configured = cudaFuncSetAttribute(
      router_fwd_kernel<NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_SMEM_BUDGET + 1024 + RT_TABLES);
  if (configured != cudaSuccess) return configured;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.split);
  cfg.blockDim = dim3(RT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = p.split;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.split > 1 ? 2 : 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, router_fwd_kernel<NG>, tmX, tmW, p);
}

cudaError_t launch_router_fwd(const RouterFwdArgs& a, cudaStream_t stream) {
  if (a.E <= 0 || a.E > kRouterMaxExperts || a.E % 8 != 0 || a.K <= 0 || a.K > kRouterMaxTopK || a.K > a.E ||
      a.H % 8 != 0 || a.n_tokens <= 0 || (a.stats != nullptr && a.workspace == nullptr))
    return cudaErrorInvalidValue;
  CUtensorMap tmX, tmW;
  RouterParams p;
  p.n_tokens = a.n_tokens;
  p.H = a.H;
  p.E = a.E;
  p.K = a.K;
  // Tiles and clusters are made smaller while they still fit one wave of SMs.  The experts are split first: every tile
  // reads the gate weights whole, at 128 experts as many bytes per k-block as the tokens of a full tile.
  const int sms = a.num_sms > 0 ? a.num_sms : 148;
  auto tiles_of = [&](int rows) { return (a.n_tokens + rows - 1) / rows; };
  p.rows = RT_BM;
  p.split = 1;
  while (p.split < 4 && a.E % (128 * p.split) == 0 && tiles_of(RT_BM) * p.split * 2 <= sms) p.split *= 2;
  while (p.rows > 16 && p.rows > 8 * p.split && tiles_of(p.rows / 2) * p.split <= sms) p.rows /= 2;
  const unsigned tiles = static_cast<unsigned>(tiles_of(p.rows));
  const int e_cta = a.E / p.split;
  p.n_chunks = (e_cta + 63) / 64;
  const int stage_bytes = RT_SUB * (p.rows * RT_BK * 2 + p.n_chunks * RT_CHUNK_BYTES);
  const int k_steps = (a.H + RT_SUB * RT_BK - 1) / (RT_SUB * RT_BK);
  int stages = RT_SMEM_BUDGET / stage_bytes;
  if (stages > RT_MAX_STAGES) stages = RT_MAX_STAGES;
  p.stages = stages < k_steps ? stages : k_steps;
  p.umma_n = ((e_cta + 15) / 16) * 16;
  int cols = 32;
  while (cols < p.umma_n) cols <<= 1;
  p.tmem_cols = cols;
  p.logits = a.logits;
  p.topk_idx = a.topk_idx;
  p.topk_w = a.topk_w;
  p.topk_idx64 = a.topk_idx64;
  p.topk_w16 = reinterpret_cast<__nv_bfloat16*>(a.topk_w_bf16);
  p.lse = a.lse;
  p.counts = a.counts;
  p.counts64 = a.counts64;
  p.mean_prob = a.mean_prob;
  p.stats = a.stats;
  p.workspace = a.workspace;
  p.status = a.status;
  p.timeout_ns = a.timeout_ns ? a.timeout_ns : kDefaultTimeoutNs;

  cudaError_t e = make_tmap(&tmX, a.X, a.n_tokens, a.H, a.ldx, p.rows);
  if (e != cudaSuccess) return e;
  e = make_tmap(&tmW, a.Wg, a.H, a.E, a.E, 64);
  if (e != cudaSuccess) return e;
  const int tile_bytes = p.rows * rt_row_stride(rt_groups(a.E)) * 4;
  const int ring = p.stages * stage_bytes;
  int smem = (ring > tile_bytes ? ring : tile_bytes) + 1024 + RT_TABLES;
  // an MMA reads 128 rows of A whatever the tile's rows: the last stage's must end inside this CTA's shared memory
  const int reach = (p.stages * RT_SUB - 1) * p.rows * RT_BK * 2 + RT_BM * RT_BK * 2 + 1024;
  if (smem < reach) smem = reach;
  switch (rt_groups(a.E)) {
    case 1: return launch_router_variant<1>(tmX, tmW, p, tiles, smem, stream);
    case 2: return launch_router_variant<2>(tmX, tmW, p, tiles, smem, stream);
    case 4: return launch_router_variant<4>(tmX, tmW, p, tiles, smem, stream);
    default: return launch_router_variant<8>(tmX, tmW, p, tiles, smem, stream);
  }
}

cudaError_t launch_router_bwd(const RouterBwdArgs& a, cudaStream_t stream) {
  const auto off16 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 != 0; };  // 16-byte vectors throughout
  if (a.E <= 0 || a.E > kRouterMaxExperts || a.E % 8 != 0 || a.K <= 0 || a.K > kRouterMaxTopK || a.n_tokens <= 0 ||
      off16(a.logits) || off16(a.counts) || off16(a.grad_logits_f32) || off16(a.grad_logits_bf16))
    return cudaErrorInvalidValue;
  const unsigned grid = static_cast<unsigned>((a.n_tokens * 8 + 255) / 256);
  return launch_chained(router_bwd_kernel, grid, 256, 0, stream, a);
}

}  // namespace cmoe
