// Two-SM variant of the tcgen05 GEMM (`tcgen05.mma.cta_group::2`): a cluster of two CTAs on neighbouring SMs works on
// one 256 x 256 output tile.  Each CTA loads its own 128 rows of A and its own 128-column half of B (ordinary TMA
// loads, every CTA its own, no cluster broadcast), the leader CTA issues one MMA per 16 k that reads both CTAs'
// shared memory and accumulates 128 rows in each CTA's tensor memory.  Per CTA and k-block that is 32 KiB of
// operands for 128 x 256 x 64 multiply-adds instead of the 48 KiB of the one-CTA kernel, so the L2 -> SM traffic per
// FLOP drops by a third and six stages fit where four did.
//
// Scope: dense GEMMs, the grouped-K weight-gradient GEMMs, and the grouped-by-rows expert GEMMs with plain and SwiGLU
// results (there a pair takes two neighbouring 128-row tiles of one expert; where an expert has an odd number of tiles
// its last pair computes and discards a half).  The row pull, the scatter and unaligned results stay on the one-CTA
// kernel in gemm.cu.  The host side sends every launch that qualifies here (`CMOE_GEMM_2CTA=0` keeps them on the
// one-CTA kernel).
// What bounds it: the tensor pipe at the clock that the power limit leaves (1.55 GHz of 1.96 in a capture of the expert
// GEMMs; pipe active 78 - 84 % of the cycles), so what counts is operand traffic per FLOP and evenly filled SMs.
// The single threads that load and issue matter as much: a k-block is 512 cycles of MMAs, and an issue loop that rebuilt
// its descriptors under a `lane == 0` branch needed about 590 (the elected form 250 to 340); a load takes its thread
// 100 to 200 cycles, so A and B have a warp each.  LM-head GEMMs of 4096 rows, H 2048, 50304 columns, before / after:
// forward 549 / 509 us, token gradient 568 / 550, weight gradient 600 / 549.
// Measured on a B200: dense 8192^3 1543 TFLOP/s against 1407 for the one-CTA kernel (cuBLAS in the same run: 1707),
// grouped weight gradient with fp32 accumulation 1352 against 1144 (both with the slower issue loop); expert layer of
// 64 experts, 2048 rows each, H 2048, F 1024, one-CTA kernel / this one / with the faster issue loop: first GEMM
// 869 / 823 / 781 us, second 475 / 436 / 413, gradient of the activation 513 / 482 / 457 (two groups of epilogue warps;
// 497 with one, slower loop), gradient of the tokens 884 / 838 / 824.
//
// CTA layout (224 threads, 352 with two epilogue groups): warp 0 TMA loads of A, the last warp those of B, warp 1 TMEM
// allocation (both CTAs) + MMA issue (leader only), the others epilogue of this CTA's 128 rows.  Barriers:
//   full[s]   in the leader: two arrivals (A, B) with the byte counts of both CTAs' loads, which complete on it
//   empty[s]  in each CTA: the leader's MMA commits to its own and to the peer's barrier
//   tfull[a]  in each CTA: committed by the leader to both when an accumulator is complete
//   tempty[a] in the leader: the epilogue threads of both CTAs
// Every wait is bounded as in gemm.cu; a wait that runs out ends the kernel normally with a status code.
#include "gemm.cuh"

#include "common.cuh"
#include "launch.h"
#include "swiglu_epilogue.cuh"
#include "tensor_maps.h"

namespace cmoe {

namespace {

constexpr int T_BM = 256;   // tile rows (128 per CTA)
constexpr int T_BN = 256;   // tile columns (each CTA loads 128 of B's rows / columns)
constexpr int T_BK = 64;
constexpr int T_A_BYTES = 128 * T_BK * 2;  // 16 KiB
constexpr int T_B_BYTES = 128 * T_BK * 2;  // 16 KiB
constexpr int T_STAGE_BYTES = T_A_BYTES + T_B_BYTES;
constexpr int T_CHUNK_BYTES = 64 * T_BK * 2;  // one 64 x 64 bf16 box of an MN-major operand
constexpr int T_STAGING_BUF = 128 * 128;
constexpr int T_STAGING = 2 * T_STAGING_BUF;  // per group of four epilogue warps
constexpr int T_MAX_GROUPS = 2;
constexpr int T_TMEM_COLS = 512;
// one group of epilogue warps leaves room for six stages, two groups for five
__host__ __device__ constexpr int t_stages(int groups) { return groups == 1 ? 6 : 5; }
__host__ __device__ constexpr int t_threads(int groups) { return 96 + 128 * groups; }
__host__ __device__ constexpr int t_smem(int groups) {
  return t_stages(groups) * T_STAGE_BYTES + groups * T_STAGING + 1024 + 256;
}
constexpr int T_EPI_FIRST = 64;

struct K2Params {
  int mode, M, N, K, groups;
  int a_mn, b_mn;
  const int* group_offsets;
  int k_chunk, k_rows;  // regular groups of k_chunk rows instead of group_offsets
  const int* tile_group;  // grouped by rows: expert of a 128-row tile, pairs of such tiles, their number
  const int* pair_tile;
  const int* num_pairs;
  int b_group_rows, split_n;
  int band;           // row tiles walked together
  const int* group_order;  // grouped by K: the groups, longest first
  int cols_per_tile;  // output columns of a tile (256; SwiGLU forward 128: gate in one CTA's half of B, up in the other's)
  int b_once;         // B is read once
  int b_early;        // B does not depend on the kernel before this one
  int has_aux;        // SwiGLU forward: gate|up is stored too
  int d_fp32, reduce;  // reduce: TMA reduce-add (fp32 accumulate) instead of store
  float2* row_stats;           // dense: softmax statistics of the rows
  int* status;
  unsigned long long timeout_ns;
};

struct Tile2 {
  int m0, n0, group, a_k0, k_blocks;
  int b_n, b_k0;  // this CTA's half of B: first N index, first K index
  bool lone;      // only the first CTA has rows
};

// `ahead`: called by the warp that does not wait for the predecessor
__device__ __forceinline__ Tile2 decode2(const K2Params& p, int t, int m_tiles, int n_tiles, int cta, bool ahead = false) {
  Tile2 ti;
  int g = 0;
  if (p.mode == GEMM_GROUPED_K) {
    g = t / (m_tiles * n_tiles);
    t -= g * m_tiles * n_tiles;
    if (p.group_order != nullptr) g = p.group_order[g];
  }
  const int band = t / (p.band * n_tiles);
  const int r = t - band * p.band * n_tiles;
  const int band_rows = min(p.band, m_tiles - band * p.band);
  const int mt = band * p.band + r % band_rows;
  ti.m0 = mt * T_BM;
  ti.n0 = (r / band_rows) * p.cols_per_tile;
  ti.b_n = ti.n0 + cta * 128;
  ti.a_k0 = ti.b_k0 = 0;
  ti.lone = false;
  ti.k_blocks = (p.K + T_BK - 1) / T_BK;
  if (p.mode == GEMM_GROUPED_K) {
    const int r0 = p.k_chunk > 0 ? min(g * p.k_chunk, p.k_rows) : p.group_offsets[g];
    const int r1 = p.k_chunk > 0 ? min((g + 1) * p.k_chunk, p.k_rows) : p.group_offsets[g + 1];
    ti.a_k0 = ti.b_k0 = r0;
    ti.k_blocks = (r1 - r0 + T_BK - 1) / T_BK;
  } else if (p.mode == GEMM_GROUPED_M) {
    const int v = ahead ? load_ahead_of_wait(p.pair_tile + mt) : p.pair_tile[mt];
    ti.m0 = (v >> 1) * 128;
    ti.lone = (v & 1) != 0;
    g = ahead ? load_ahead_of_wait(p.tile_group + (v >> 1)) : p.tile_group[v >> 1];
    if (p.b_mn) {
      ti.b_k0 = g * p.b_group_rows;
    } else {
      ti.b_n = g * p.b_group_rows + (p.split_n ? ti.n0 + cta * p.split_n : ti.b_n);
    }
  }
  ti.group = g;
  return ti;
}

// The tile of cluster c in the round of tiles that starts at r0 (one per cluster).  With the groups sorted by length
// the rounds go back and forth, so that a cluster which got the longest tile of one round gets the shortest of the next.
__device__ __forceinline__ int tile_of_round(const K2Params& p, int r0, int c, int n_clusters) {
  return p.group_order != nullptr && ((r0 / n_clusters) & 1) != 0 ? r0 + n_clusters - 1 - c : r0 + c;
}

// ---- cluster / two-SM PTX -------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load of this CTA's operand piece whose bytes are counted on a barrier that may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tmap, uint32_t bar_cluster_addr,
                                                 int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair_policy(void* smem_dst, const CUtensorMap* tmap, uint32_t bar_cluster_addr,
                                                        int x, int y, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_cluster_addr), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrives once on the barrier at this shared-memory offset in both CTAs when all MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_both(uint32_t smem_addr) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void umma_bf16_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Adds 64 values of a row, packed in bf16 pairs of which the first `live` columns exist, to its running maximum and sum of
// exp(v - maximum).  A row of minus infinities only has the sum 0.
__device__ __forceinline__ void add_to_stats(const uint32_t (&v)[32], int live, float& mx, float& sum) {
  float m = mx;
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (2 * j < live) m = fmaxf(m, fmaxf(__uint_as_float(v[j] << 16), __uint_as_float(v[j] & 0xffff0000u)));
  const float base = m == -INFINITY ? 0.f : m;
  sum *= __expf(mx - base);
  mx = m;
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (2 * j < live)
      sum += __expf(__uint_as_float(v[j] << 16) - base) + __expf(__uint_as_float(v[j] & 0xffff0000u) - base);
}

// STATS: the softmax statistics of the rows are left too.  A kernel of its own: the registers and branches that they take
// in the epilogue cost every other bf16 result 0.3 to 2 % (4096 x 4096 result rows of 256 terms 30.4 / 31.0 us).
template <int EPI, int GROUPS, bool STATS = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(t_threads(GROUPS), 1)
gemm2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
             const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmE, const K2Params p) {
  constexpr int T_STAGES = t_stages(GROUPS);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + T_STAGES * T_A_BYTES;
  uint8_t* stg = smem + T_STAGES * T_STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T_STAGES * T_STAGE_BYTES + GROUPS * T_STAGING);
  uint64_t* full_bar = bars;                    // [T_STAGES]  (used in the leader)
  uint64_t* empty_bar = bars + T_STAGES;        // [T_STAGES]
  uint64_t* tfull_bar = bars + 2 * T_STAGES;    // [2]
  uint64_t* tempty_bar = bars + 2 * T_STAGES + 2;  // [2]       (used in the leader)
  uint64_t* gfull_bar = bars + 2 * T_STAGES + 4;   // [GROUPS][2] saved gate|up pieces (SwiGLU backward)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * T_STAGES + 4 + 2 * T_MAX_GROUPS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();  // 0: leader (issues the MMAs), 1: peer
  const bool leader = cta == 0;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < T_STAGES; ++s) {
      mbar_init(&full_bar[s], 2);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 256 * GROUPS);
    }
    for (int a = 0; a < 2 * GROUPS; ++a) mbar_init(&gfull_bar[a], 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmD);
    if (EPI != EPI_STORE) tma_prefetch_desc(&tmE);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, T_TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anybody signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  WaitCtx wc;
  wc.abort_flag = abort_flag;
  wc.status = p.status;
  wc.timeout_ns = p.timeout_ns;

  // what the kernel before this one wrote (or still reads) is touched behind this line only; weights that nobody writes
  // and the row plan, which is older than that kernel, may be loaded ahead of it
  const bool ahead = p.b_early && warp == 2 + 4 * GROUPS;
  if (!ahead) {
    chain_wait();
    chain_trigger();
  }

  const int m_tiles = p.mode == GEMM_GROUPED_M ? (ahead ? load_ahead_of_wait(p.num_pairs) : *p.num_pairs) : (p.M + T_BM - 1) / T_BM;
  const int n_tiles = (p.N + p.cols_per_tile - 1) / p.cols_per_tile;
  const int n_total = (p.mode == GEMM_GROUPED_K ? p.groups : 1) * m_tiles * n_tiles;
  const int cluster_id = blockIdx.x >> 1;
  const int n_clusters = gridDim.x >> 1;

  if (warp == 0 || warp == 2 + 4 * GROUPS) {
    // ------------------------------------------------------------------ TMA producers (both CTAs)
    // One warp loads A, one B: a thread needs 100 - 200 cycles to issue a load, and a k-block has two to four of them.
    if (elect_one()) {
      const bool is_a = warp == 0;
      const CUtensorMap* tm = is_a ? &tmA : &tmB;
      const bool mn = is_a ? p.a_mn != 0 : p.b_mn != 0;
      uint8_t* const dst0 = is_a ? sA : sB;
      const uint32_t fb0 = map_to_cta(smem_u32(full_bar), 0);
      const uint64_t once = l2_evict_first();
      const bool stream = !is_a && p.b_once;
      const int moff = static_cast<int>(cta) * 128;  // this CTA's rows of A
      int stage = 0;
      uint32_t phase = 0;
      for (int r0 = 0; r0 < n_total; r0 += n_clusters) {
        const int t = tile_of_round(p, r0, cluster_id, n_clusters);
        if (t >= n_total) break;  // in the last round only
        const Tile2 ti = decode2(p, t, m_tiles, n_tiles, static_cast<int>(cta), ahead);
        if (ti.k_blocks == 0) continue;
        const int x = is_a ? ti.m0 + moff : ti.b_n;
        int k = is_a ? ti.a_k0 : ti.b_k0;
        const bool skip = is_a && ti.lone;  // one CTA's rows only; the MMA reads stale ones there, which are not stored
        const uint32_t bytes = (skip ? 1 : 2) * T_A_BYTES;
        const bool load = leader || !skip;
        for (int kb = 0; kb < ti.k_blocks; ++kb, k += T_BK) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, wc, ST_TIMEOUT_SMEM_EMPTY)) break;
          const uint32_t fb = fb0 + stage * 8;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], bytes);
          uint8_t* dst = dst0 + stage * T_A_BYTES;
          if (load) {
            if (mn) {
              tma_load_2d_pair(dst, tm, fb, x, k);
              tma_load_2d_pair(dst + T_CHUNK_BYTES, tm, fb, x + 64, k);
            } else if (stream) {
              tma_load_2d_pair_policy(dst, tm, fb, k, x, once);
            } else {
              tma_load_2d_pair(dst, tm, fb, k, x);
            }
          }
          if (++stage == T_STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (*abort_flag) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    // The loop body is what one thread issues while the tensor pipe works on 512 cycles' worth of MMAs: the elected
    // thread is known to be alone (no loop over the lanes around each instruction) and the descriptors only advance.
    if (leader && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(T_BM, T_BN, p.a_mn, p.b_mn);
      const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(sA), p.a_mn ? T_CHUNK_BYTES : 16, 1024);
      const uint64_t b_desc0 = make_smem_desc_sw128(smem_u32(sB), p.b_mn ? T_CHUNK_BYTES : 16, 1024);
      const uint32_t a_kstep = (p.a_mn ? 2048u : 32u) >> 4;
      const uint32_t b_kstep = (p.b_mn ? 2048u : 32u) >> 4;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int r0 = 0; r0 < n_total; r0 += n_clusters) {
        const int t = tile_of_round(p, r0, cluster_id, n_clusters);
        if (t >= n_total) break;  // in the last round only
        const Tile2 ti = decode2(p, t, m_tiles, n_tiles, static_cast<int>(cta));
        if (ti.k_blocks == 0) continue;
        if (!mbar_wait(&tempty_bar[acc], acc_phase ^ 1u, wc, ST_TIMEOUT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * T_BN;
        for (int kb = 0; kb < ti.k_blocks; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, wc, ST_TIMEOUT_SMEM_FULL)) break;
          tc_fence_after();
          const uint64_t ad = a_desc0 + static_cast<uint32_t>(stage * (T_A_BYTES >> 4));
          const uint64_t bd = b_desc0 + static_cast<uint32_t>(stage * (T_B_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < T_BK / 16; ++k)
            umma_bf16_ss_pair(d_tmem, ad + k * a_kstep, bd + k * b_kstep, idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit_both(smem_u32(&empty_bar[stage]));  // the stage is free in both CTAs once these MMAs have read it
          if (++stage == T_STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        umma_commit_both(smem_u32(&tfull_bar[acc]));
        if (*abort_flag) break;
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (this CTA's 128 rows)
    // With two groups of four warps, a group takes every second piece of columns and has its own staging buffers.
    const int grp = GROUPS == 1 ? 0 : (warp - 2) >> 2;
    const bool issuer = threadIdx.x == T_EPI_FIRST + 128 * grp;  // of this group's TMA copies
    uint8_t* my_stg = stg + grp * T_STAGING;
    const int quad = warp & 3;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const int sw = row_in_tile & 7;
    const int gsw = (row_in_tile >> 1) & 3;  // 64-byte swizzle: 16-byte chunk j of row r sits at j ^ ((r / 2) % 4)
    const int unit_cols = EPI != EPI_STORE || p.d_fp32 ? 32 : 64;
    // one named barrier per group and piece; it carries the OR of "a wait failed / abort seen", so that all 128
    // threads leave the loop together
    auto any_failed = [&](bool bad_here) {
      int any;
      asm volatile(
          "{\n\t.reg .pred q, r;\n\tsetp.ne.s32 q, %1, 0;\n\tbar.red.or.pred r, %2, 128, q;\n\t"
          "selp.s32 %0, 1, 0, r;\n\t}"
          : "=r"(any)
          : "r"((bad_here || *abort_flag) ? 1 : 0), "r"(1 + grp)
          : "memory");
      return any != 0;
    };
    int acc = 0;
    uint32_t acc_phase = 0;
    uint32_t stage_ctr = 0;
    for (int r0 = 0; r0 < n_total; r0 += n_clusters) {
      const int t = tile_of_round(p, r0, cluster_id, n_clusters);
      if (t >= n_total) break;  // in the last round only
      const Tile2 ti = decode2(p, t, m_tiles, n_tiles, static_cast<int>(cta));
      const int row0 = ti.m0 + static_cast<int>(cta) * 128;
      const bool have_acc = ti.k_blocks != 0;
      if (!have_acc && (p.reduce || EPI != EPI_STORE)) continue;  // adding zero: nothing to do (K > 0 otherwise)
      const bool mine = p.mode == GEMM_GROUPED_M ? (leader || !ti.lone) : row0 < p.M;  // this CTA has rows
      // SwiGLU backward: asks for the saved gate and up values of a piece (128 rows x 32 columns each)
      auto gu_issue = [&](uint32_t ctr, int col) {
        const uint32_t b = ctr & 1u;
        uint8_t* dst = my_stg + b * T_STAGING_BUF;
        uint64_t* bar = &gfull_bar[2 * grp + b];
        mbar_arrive_expect_tx(bar, T_STAGING_BUF);
        tma_load_2d(dst, &tmD, bar, col, row0);
        tma_load_2d(dst + T_STAGING_BUF / 2, &tmD, bar, p.N + col, row0);
      };
      if (EPI == EPI_SWIGLU_BWD && issuer && mine && ti.n0 + grp * 32 < p.N) {
        bulk_wait_group_read<1>();  // this piece's buffer was last read by the store issued two pieces ago
        gu_issue(stage_ctr, ti.n0 + grp * 32);
      }
      float stat_max = -INFINITY, stat_sum = 0.f;
      bool ok = true;
      if (have_acc) {
        ok = mbar_wait(&tfull_bar[acc], acc_phase, wc, ST_TIMEOUT_TMEM_FULL);
        tc_fence_after();
      }
      const uint32_t t_acc = tmem_base + acc * T_BN + lane_base;
      bool any_bad = false;
      const int units = p.cols_per_tile / unit_cols;
#pragma unroll 1
      for (int u = grp; u < units; u += GROUPS) {
        const int col0 = ti.n0 + u * unit_cols;
        if (col0 >= p.N) break;  // uniform
        if (EPI == EPI_SWIGLU_BWD) {
          // every thread turns its row of the piece into dGate / dUp in place
          if (!mine) break;
          const uint32_t b = stage_ctr & 1u;
          if (issuer && u + GROUPS < units && col0 + 32 * GROUPS < p.N) {
            bulk_wait_group_read<0>();  // the store of the previous piece has read the other buffer
            gu_issue(stage_ctr + 1, col0 + 32 * GROUPS);
          }
          const bool got = mbar_wait(&gfull_bar[2 * grp + b], (stage_ctr >> 1) & 1u, wc, ST_TIMEOUT_SMEM_FULL);
          uint8_t* grow = my_stg + b * T_STAGING_BUF + row_in_tile * 64;
          if (ok && got) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(t_acc + u * 32, r);
            uint4 cg[4], cu[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              cg[j] = *reinterpret_cast<const uint4*>(grow + ((j ^ gsw) << 4));
              cu[j] = *reinterpret_cast<const uint4*>(grow + T_STAGING_BUF / 2 + ((j ^ gsw) << 4));
            }
            tmem_ld_wait();
            swiglu_bwd_math(r, cg, cu);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              *reinterpret_cast<uint4*>(grow + ((j ^ gsw) << 4)) = cg[j];
              *reinterpret_cast<uint4*>(grow + T_STAGING_BUF / 2 + ((j ^ gsw) << 4)) = cu[j];
            }
          }
          fence_proxy_async_smem();
          any_bad = any_failed(!ok || !got);
          if (any_bad) break;
          if (issuer) {
            tma_store_3d(&tmE, my_stg + b * T_STAGING_BUF, col0, 0, row0);                      // dGate
            tma_store_3d(&tmE, my_stg + b * T_STAGING_BUF + T_STAGING_BUF / 2, col0, 1, row0);  // dUp
            bulk_commit_group();
          }
          ++stage_ctr;
          continue;
        }
        if (EPI == EPI_SWIGLU_FWD) {
          // accumulator columns [0, 128) = gate, [128, 256) = up: h, gate and up leave as three pieces of 128 rows x
          // 64 bytes out of one staging area; two barriers per piece (area free, area filled)
          if (!mine) break;
          uint8_t* hrow = my_stg + row_in_tile * 64;
          uint32_t ph[16], pg[16], pu[16];
          if (ok) {
            uint32_t rg[32], ru[32];
            tmem_ld_32x32b_x32(t_acc + u * 32, rg);
            tmem_ld_32x32b_x32(t_acc + 128 + u * 32, ru);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float g0 = __uint_as_float(rg[2 * j]), g1 = __uint_as_float(rg[2 * j + 1]);
              const float u0 = __uint_as_float(ru[2 * j]), u1 = __uint_as_float(ru[2 * j + 1]);
              ph[j] = pack_bf16x2(g0 * sigmoidf_fast(g0) * u0, g1 * sigmoidf_fast(g1) * u1);
              pg[j] = pack_bf16x2(g0, g1);
              pu[j] = pack_bf16x2(u0, u1);
            }
          }
          if (issuer) bulk_wait_group_read<0>();  // the stores of the previous piece have read the area
          any_bad = any_failed(!ok);
          if (any_bad) break;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int o = (j ^ gsw) << 4;
            *reinterpret_cast<uint4*>(hrow + o) = make_uint4(ph[4 * j], ph[4 * j + 1], ph[4 * j + 2], ph[4 * j + 3]);
            if (p.has_aux) {
              *reinterpret_cast<uint4*>(hrow + T_STAGING_BUF / 2 + o) =
                  make_uint4(pg[4 * j], pg[4 * j + 1], pg[4 * j + 2], pg[4 * j + 3]);
              *reinterpret_cast<uint4*>(hrow + T_STAGING_BUF + o) =
                  make_uint4(pu[4 * j], pu[4 * j + 1], pu[4 * j + 2], pu[4 * j + 3]);
            }
          }
          fence_proxy_async_smem();
          asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
          if (issuer) {
            tma_store_3d(&tmD, my_stg, col0, row0, 0);
            if (p.has_aux) {
              tma_store_3d(&tmE, my_stg + T_STAGING_BUF / 2, col0, 0, row0);  // gate half
              tma_store_3d(&tmE, my_stg + T_STAGING_BUF, col0, 1, row0);      // up half
            }
            bulk_commit_group();
          }
          continue;
        }
        uint8_t* buf = my_stg + (stage_ctr & 1) * T_STAGING_BUF;
        uint8_t* myrow = buf + row_in_tile * 128;
        if (ok) {
          if (p.d_fp32) {
            uint32_t r[32];
            if (have_acc) {
              tmem_ld_32x32b_x32(t_acc + u * 32, r);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<uint4*>(myrow + ((j ^ sw) << 4)) =
                  make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          } else {
            uint32_t r0[32], r1[32];
            if (have_acc) {
              tmem_ld_32x32b_x32(t_acc + u * 64, r0);
              tmem_ld_32x32b_x32(t_acc + u * 64 + 32, r1);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) r0[j] = r1[j] = 0u;
            }
            uint32_t v[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              v[j] = pack_bf16x2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1]));
              v[16 + j] = pack_bf16x2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<uint4*>(myrow + ((j ^ sw) << 4)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            if (STATS) {
              const int live = p.N - col0;
              if (live >= 64)
                add_to_stats(v, 64, stat_max, stat_sum);
              else
                add_to_stats(v, live, stat_max, stat_sum);
            }
          }
        }
        fence_proxy_async_smem();
        if (issuer) bulk_wait_group_read<0>();
        any_bad = any_failed(!ok);
        if (any_bad) break;
        if (issuer && mine) {
          const int zgrp = (p.mode == GEMM_GROUPED_K) ? ti.group : 0;
          if (p.reduce)
            tma_reduce_add_3d(&tmD, buf, col0, row0, zgrp);
          else
            tma_store_3d(&tmD, buf, col0, row0, zgrp);
          bulk_commit_group();
        }
        ++stage_ctr;
      }
      if (STATS && row0 + row_in_tile < p.M)
        p.row_stats[static_cast<long long>(row0 + row_in_tile) * n_tiles + ti.n0 / T_BN] = make_float2(stat_max, stat_sum);
      if (have_acc) {
        // the leader's MMA warp may reuse this accumulator once all epilogue threads of the pair have read it
        tc_fence_before();
        mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[acc]), 0));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
      if (any_bad) break;
    }
    if (issuer) bulk_wait_group<0>();
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while the other may still touch it
  if (warp == 1) {
    if (*abort_flag) {
      for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, T_TMEM_COLS);
  }
}

}  // namespace

bool gemm_2cta_supported(const GemmArgs& a) {
  if (a.scatter_row_slot != nullptr || a.pull_row_slot != nullptr || a.ready_flags != nullptr || a.tile_rows != nullptr ||
      a.tile_n != 0)
    return false;
  if (a.N % 8 != 0 || a.N <= 0) return false;
  const auto aligned = [](const void* ptr, long long ld, long long es) {
    return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0 && (ld * es) % 16 == 0;
  };
  const long long es = a.d_fp32 ? 4 : 2;
  long long gstride = static_cast<long long>(a.M) * a.ldd;
  if (a.mode == GEMM_DENSE) {
    if (a.a_mn || a.M <= 0 || (a.row_stats != nullptr && (a.d_fp32 || a.accumulate || a.epilogue != EPI_STORE))) return false;
  } else if (a.mode == GEMM_GROUPED_K) {
    if (!(a.a_mn && a.b_mn) || (a.group_offsets == nullptr && (a.k_chunk <= 0 || a.k_chunk % 64 != 0)) || a.M <= 0)
      return false;
    gstride = a.d_group_stride;
  } else {
    if (a.pair_tile == nullptr || a.a_mn || a.K <= 0 || a.accumulate) return false;
    gstride = 0;
  }
  if (a.epilogue != EPI_STORE) {
    if (a.mode != GEMM_GROUPED_M || a.d_fp32 || !aligned(a.D, a.ldd, 2)) return false;
    if (a.epilogue == EPI_SWIGLU_FWD)
      return !a.b_mn && a.split_n > 0 && a.ldd >= a.N &&
             (a.aux_out == nullptr || (aligned(a.aux_out, a.ld_aux_out, 2) && a.ld_aux_out >= 2LL * a.N));
    return a.epilogue == EPI_SWIGLU_BWD && a.aux_in != nullptr && aligned(a.aux_in, a.ld_aux_in, 2) &&
           a.ld_aux_in >= 2LL * a.N && a.ldd >= 2LL * a.N;
  }
  if (a.accumulate && !a.d_fp32) return false;
  return aligned(a.D, a.ldd, es) && (gstride * es) % 16 == 0 && a.ldd >= a.N;
}

template <int EPI, int GROUPS, bool STATS = false>
static cudaError_t launch_pairs(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmD,
                                const CUtensorMap& tmE, const K2Params& kp, long long clusters, cudaStream_t stream) {
  static const cudaError_t configured =
      cudaFuncSetAttribute(gemm2_kernel<EPI, GROUPS, STATS>, cudaFuncAttributeMaxDynamicSharedMemorySize, t_smem(GROUPS));
  if (configured != cudaSuccess) return configured;
  return launch_chained(gemm2_kernel<EPI, GROUPS, STATS>, static_cast<unsigned>(2 * clusters), t_threads(GROUPS),
                        t_smem(GROUPS), stream, tmA, tmB, tmD, tmE, kp);
}

cudaError_t launch_gemm_2cta(const GemmArgs& a, cudaStream_t stream) {
  if (!gemm_2cta_supported(a)) return cudaErrorInvalidValue;
  CUtensorMap tmA, tmB, tmD, tmE;
  cudaError_t e = make_tmap(&tmA, a.A, a.a_rows, a.a_cols, a.a_ld, a.a_mn ? 64 : 128);
  if (e != cudaSuccess) return e;
  e = make_tmap(&tmB, a.B, a.b_rows, a.b_cols, a.b_ld, a.b_mn ? 64 : 128);
  if (e != cudaSuccess) return e;
  const long long groups = a.mode == GEMM_GROUPED_K ? a.groups : 1;
  const long long d_rows = a.mode == GEMM_GROUPED_M ? a.a_rows : a.M;
  const long long gstride = a.mode == GEMM_GROUPED_K ? a.d_group_stride : d_rows * a.ldd;
  tmE = tmA;  // placeholder where the epilogue has no second map
  if (a.epilogue == EPI_STORE) {
    e = make_tmap_out(&tmD, a.D, a.d_fp32, groups, d_rows, a.N, a.ldd, gstride);
  } else if (a.epilogue == EPI_SWIGLU_FWD) {
    e = make_tmap_out(&tmD, a.D, 0, 1, d_rows, a.N, a.ldd, gstride, 64);
    if (e == cudaSuccess && a.aux_out != nullptr) e = make_tmap_halves(&tmE, a.aux_out, d_rows, a.N, a.ld_aux_out);
  } else {
    e = make_tmap(&tmD, a.aux_in, d_rows, 2LL * a.N, a.ld_aux_in, 128, 32);
    if (e == cudaSuccess) e = make_tmap_halves(&tmE, a.D, d_rows, a.N, a.ldd);
  }
  if (e != cudaSuccess) return e;

  K2Params kp;
  kp.mode = a.mode;
  kp.M = a.M;
  kp.N = a.N;
  kp.K = a.K;
  kp.groups = a.groups;
  kp.a_mn = a.a_mn;
  kp.b_mn = a.b_mn;
  kp.group_offsets = a.group_offsets;
  kp.k_chunk = a.k_chunk;
  kp.k_rows = static_cast<int>(a.a_rows);
  kp.tile_group = a.tile_group;
  kp.pair_tile = a.pair_tile;
  kp.num_pairs = a.num_pairs;
  kp.b_group_rows = static_cast<int>(a.b_group_rows);
  kp.split_n = a.epilogue == EPI_SWIGLU_FWD ? a.split_n : 0;
  kp.group_order = a.mode == GEMM_GROUPED_K ? a.group_order : nullptr;
  // A band of row tiles is walked column by column, and B is read once per band: eight row tiles where B is the larger
  // operand and a group has that many, four otherwise (a band across several groups reads more of B at a time).
  // 8 experts x 2048 rows, H 4096, F 14336: first GEMM 3260 -> 3110 us, gradient of the activation 1695 -> 1630;
  // 833 rows per expert: 755 -> 760.
  const long long group_rows = a.mode == GEMM_GROUPED_M ? a.rows_per_group : a.M;
  const long long b_extent = a.epilogue == EPI_SWIGLU_FWD ? 2LL * a.N : a.N;
  kp.band = b_extent > group_rows && group_rows >= 8 * T_BM ? 8 : 4;
  kp.cols_per_tile = a.epilogue == EPI_SWIGLU_FWD ? 128 : T_BN;
  kp.b_once = a.b_once;
  kp.b_early = a.b_early;
  kp.has_aux = a.aux_out != nullptr;
  kp.d_fp32 = a.d_fp32;
  kp.reduce = a.accumulate;
  kp.row_stats = a.row_stats;
  kp.status = a.status;
  kp.timeout_ns = a.timeout_ns ? a.timeout_ns : kDefaultTimeoutNs;

  int num_sms = a.num_sms;
  if (num_sms <= 0) {
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
  }
  // grouped by rows: an expert's last pair may have one tile only, so up to max_m_tiles pairs
  const long long m_tiles = a.mode == GEMM_GROUPED_M ? a.max_m_tiles : (a.M + T_BM - 1) / T_BM;
  const long long tiles = m_tiles * ((a.N + kp.cols_per_tile - 1) / kp.cols_per_tile) * groups;
  if (tiles <= 0) return cudaSuccess;
  const long long clusters = tiles < num_sms / 2 ? tiles : num_sms / 2;
  switch (a.epilogue) {
    case EPI_STORE:
      return a.row_stats != nullptr ? launch_pairs<EPI_STORE, 1, true>(tmA, tmB, tmD, tmE, kp, clusters, stream)
                                    : launch_pairs<EPI_STORE, 1>(tmA, tmB, tmD, tmE, kp, clusters, stream);
    case EPI_SWIGLU_FWD:
      return launch_pairs<EPI_SWIGLU_FWD, 1>(tmA, tmB, tmD, tmE, kp, clusters, stream);
    default:
      return launch_pairs<EPI_SWIGLU_BWD, 2>(tmA, tmB, tmD, tmE, kp, clusters, stream);
  }
}

}  // namespace cmoe
