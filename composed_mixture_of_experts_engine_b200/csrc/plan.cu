// Expert-sorted row plan of the MoE layer (see ops.cuh for what it produces): ranks every (token, k) slot within its
// expert, in slot order and without atomics on the order.
// Reference counterpart: argsort / repeat_interleave of the MoE layer (pkg/distributed/moe_layer.py:309-353) and its
// capacity dropping (moe_layer.py:64-155).
//
// What bounds it: latency.  The slots are a few hundred KiB at most, so the time is the number of dependent launches
// and of dependent passes inside them.
//   * up to 8192 slots: one launch of one CTA, 32 warps that each rank 256 slots;
//   * more: a counting launch (histogram per unit of slots), then one launch whose CTAs each add up the histograms of
//     the units before theirs (a few KiB out of L2, redundantly, which is cheaper than a launch or a last-CTA hand-over
//     in between), derive the expert offsets and rank their slots;
//   * only where units x bins exceed 16384 words a scan launch replaces the redundant sums;
//   * few slots over thousands of bins: one CTA with two words per bin, since eight warps' counts of every bin would be
//     more work to clear and add up than the slots are.
//     One call, eight warps' counts / this: 400 tokens top-8 of 1024 experts with capacity 230 / 83 us, 512 x 8 of 4500
//     experts 232 / 124, 100 x 2 of 40000 1392 / 462.
// The first form took two memsets and three launches, one of them a single CTA whose first thread walked the experts
// through global memory: 22.8 us of kernels for 64 tokens x top-8 of 64 experts, 41 us for 16384 tokens.
#include "ops.cuh"

#include "common.cuh"
#include "launch.h"

namespace cmoe {

namespace {

constexpr int kCountThreads = 256;
constexpr int kWarpsMulti = 8;
constexpr int kWarpsSingle = 32;
constexpr int kSingleSlots = 8192;
constexpr int kRedundantWords = 16384;
constexpr int kSparseSlots = 4096;
constexpr int kSmemLimit = 200 * 1024;

__device__ __forceinline__ int plan_bin(const MoePlanArgs& a, long long slot) {
  const int e = a.topk_idx[slot] - a.expert_lo;
  if (e < 0 || e >= a.n_local) return -1;
  return a.per_k_bins ? e * a.K + static_cast<int>(slot % a.K) : e;
}

// hist[unit][bin]; also clears the row -> slot table
__global__ void __launch_bounds__(kCountThreads) plan_count_kernel(const MoePlanArgs a, int nbins, int unit_slots,
                                                                   int in_smem) {
  chain_wait();
  chain_trigger();
  extern __shared__ int plan_smem[];
  int* hist = a.scratch + static_cast<long long>(blockIdx.x) * nbins;
  int* h = in_smem ? plan_smem : hist;
  for (int b = threadIdx.x; b < nbins; b += kCountThreads) h[b] = 0;
  for (long long r = blockIdx.x * static_cast<long long>(kCountThreads) + threadIdx.x; r < a.cap_rows;
       r += static_cast<long long>(gridDim.x) * kCountThreads)
    a.row_slot[r] = -1;
  __syncthreads();
  const long long s0 = static_cast<long long>(blockIdx.x) * unit_slots;
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int i = threadIdx.x; i < unit_slots; i += kCountThreads) {  // whole warps: unit_slots is a multiple of 1024
    const long long slot = s0 + i;
    const int bin = slot < a.n_slots ? plan_bin(a, slot) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, bin);
    if (bin >= 0 && (peers & ((1u << lane) - 1u)) == 0u) atomicAdd(h + bin, __popc(peers));
  }
  if (in_smem) {
    __syncthreads();
    for (int b = threadIdx.x; b < nbins; b += kCountThreads) hist[b] = h[b];
  }
}

// In place: hist[unit][bin] -> sum over the units before it; total[bin] behind the histograms.  A CTA takes 32 bins,
// its 32 warps a chunk of the units each.
__global__ void __launch_bounds__(1024) plan_scan_kernel(const MoePlanArgs a, int nbins, int n_units) {
  chain_wait();
  chain_trigger();
  __shared__ int part[32][33];
  int* hist = a.scratch;
  int* total = a.scratch + static_cast<long long>(n_units) * nbins;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = blockIdx.x * 32 + lane;
  const int per = (n_units + 31) / 32;
  const int u0 = min(n_units, w * per), u1 = min(n_units, u0 + per);
  int sum = 0;
  if (b < nbins)
#pragma unroll 8
    for (int u = u0; u < u1; ++u) sum += hist[static_cast<long long>(u) * nbins + b];
  part[w][lane] = sum;
  __syncthreads();
  int run = 0;
  for (int q = 0; q < w; ++q) run += part[q][lane];
  if (b < nbins) {
#pragma unroll 8
    for (int u = u0; u < u1; ++u) {
      const int c = hist[static_cast<long long>(u) * nbins + b];
      hist[static_cast<long long>(u) * nbins + b] = run;
      run += c;
    }
    if (w == 31) total[b] = run;
  }
}

// int words of working storage of one CTA of the ranking kernel: warp counts, slots before this unit, totals, first
// row of every bin, first row and first tile pair of every expert
__host__ __device__ inline long long rank_words(int warps, int nbins, int n_local) {
  return (static_cast<long long>(warps) + 3) * nbins + 2 * (n_local + 1);
}

// SINGLE: one CTA does everything.  Otherwise CTA u ranks the slots of unit u; `prescanned` says that
// plan_scan_kernel has run.  `work` is this launch's working storage in global memory, one piece per CTA, where shared
// memory would not hold it (thousands of bins); nullptr: shared memory.
template <int WARPS, bool SINGLE>
__global__ void __launch_bounds__(WARPS * 32) plan_rank_kernel(const MoePlanArgs a, int nbins, int unit_slots,
                                                               int n_units, int prescanned, int* work) {
  chain_wait();
  chain_trigger();
  extern __shared__ int plan_smem[];
  constexpr int T = WARPS * 32;
  int* s_warp = work != nullptr ? work + blockIdx.x * rank_words(WARPS, nbins, a.n_local) : plan_smem;  // [WARPS][nbins]
  int* s_pre = s_warp + WARPS * nbins;  // slots of the bin in units before this one
  int* s_tot = s_pre + nbins;           // all slots of the bin
  int* s_base = s_tot + nbins;          // first row of the bin
  int* s_goff = s_base + nbins;         // [n_local + 1] first row of the expert
  int* s_pair = s_goff + a.n_local + 1; // [n_local + 1] first pair of its tiles
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int unit = blockIdx.x;
  const unsigned below = (1u << lane) - 1u;

  for (int i = tid; i < (WARPS + 2) * nbins; i += T) s_warp[i] = 0;
  if (SINGLE)
    for (long long r = tid; r < a.cap_rows; r += T) a.row_slot[r] = -1;
  __syncthreads();

  // counts of this warp's range of slots
  const int warp_slots = unit_slots / WARPS;
  const long long s0 = static_cast<long long>(unit) * unit_slots + warp * warp_slots;
  int* mine = s_warp + warp * nbins;
  // (the expert numbers of up to eight rounds of 32 slots are fetched together)
  int bins[8];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = i0 + q * 32;
      const long long slot = s0 + i + lane;
      bins[q] = i < warp_slots && slot < a.n_slots ? plan_bin(a, slot) : -1;
    }
  };
  for (int i0 = 0; i0 < warp_slots; i0 += 256) {
    fetch(i0);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int bin = bins[q];
      const unsigned peers = __match_any_sync(0xffffffffu, bin);
      if (bin >= 0 && (peers & below) == 0u) mine[bin] += __popc(peers);
      __syncwarp();
    }
  }
  // counts of the other units
  if (!SINGLE) {
    const int* hist = a.scratch;
    if (prescanned) {
      const int* total = hist + static_cast<long long>(n_units) * nbins;
      for (int b = tid; b < nbins; b += T) {
        s_pre[b] = hist[static_cast<long long>(unit) * nbins + b];
        s_tot[b] = total[b];
      }
    } else {
      // thread = (bin, range of units)
      const int lanes_b = min(nbins, T);
      const int ranges = T / lanes_b, range = tid / lanes_b;
      if (range < ranges) {
        const int per = (n_units + ranges - 1) / ranges;
        const int u0 = min(n_units, range * per), u1 = min(n_units, u0 + per);
        for (int b = tid - range * lanes_b; b < nbins; b += lanes_b) {
          int before = 0, all = 0;
#pragma unroll 8
          for (int u = u0; u < u1; ++u) {
            const int c = hist[static_cast<long long>(u) * nbins + b];
            all += c;
            before += u < unit ? c : 0;
          }
          atomicAdd(s_pre + b, before);
          atomicAdd(s_tot + b, all);
        }
      }
    }
  }
  __syncthreads();
  // per bin: exclusive prefix over the warps
  for (int b = tid; b < nbins; b += T) {
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < WARPS; ++w) {
      const int c = s_warp[w * nbins + b];
      s_warp[w * nbins + b] = run;
      run += c;
    }
    if (SINGLE) s_tot[b] = run;
    if (a.capacity > 0) {
      const int t = SINGLE ? run : s_tot[b];
      s_tot[b] = min(t, a.capacity);
    }
  }
  __syncthreads();
  // expert offsets: 128-row-padded exclusive prefix over the experts (one warp), clipped to the buffer
  const int kb = a.per_k_bins ? a.K : 1;
  const int cap128 = static_cast<int>(a.cap_rows / 128 * 128);
  if (warp == 0) {
    long long carry = 0;
    int pair_carry = 0;
    for (int e0 = 0; e0 < a.n_local; e0 += 32) {
      const int e = e0 + lane;
      int cnt = 0;
      if (e < a.n_local)
        for (int k = 0; k < kb; ++k) cnt += s_tot[e * kb + k];
      const int padded = (cnt + 127) / 128 * 128;
      int incl = padded;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const long long raw = carry + incl - padded;
      const int off = raw < cap128 ? static_cast<int>(raw) : cap128;
      const int pairs = ((raw + padded < cap128 ? static_cast<int>(raw) + padded : cap128) - off + 255) / 256;
      int pincl = pairs;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pincl, o);
        if (lane >= o) pincl += v;
      }
      if (e < a.n_local) {
        s_goff[e] = off;
        s_pair[e] = pair_carry + pincl - pairs;
        int base = off;
        for (int k = 0; k < kb; ++k) {
          s_base[e * kb + k] = base;
          base += s_tot[e * kb + k];
        }
        if (unit == 0) {
          // rows that do not fit the buffer are dropped below (and counted in `overflow`)
          const long long room = a.cap_rows - off;
          a.counts_kept[e] = cnt > room ? static_cast<int>(room > 0 ? room : 0) : cnt;
          a.group_offsets[e] = off;
        }
      }
      carry += __shfl_sync(0xffffffffu, incl, 31);
      pair_carry += __shfl_sync(0xffffffffu, pincl, 31);
    }
    if (lane == 0) {
      const int off = carry < cap128 ? static_cast<int>(carry) : cap128;
      s_goff[a.n_local] = off;
      if (unit == 0) {
        a.group_offsets[a.n_local] = off;
        *a.num_m_tiles = off / 128;
        if (a.num_pairs != nullptr) *a.num_pairs = pair_carry;
      }
    }
  }
  __syncthreads();
  // destination row of every slot
  for (int i0 = 0; i0 < warp_slots; i0 += 256) {
    if (warp_slots > 256) fetch(i0);  // otherwise still at hand
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = i0 + q * 32;
      const long long slot = s0 + i + lane;
      const int bin = bins[q];
      const unsigned peers = __match_any_sync(0xffffffffu, bin);
      int row = -1;
      if (bin >= 0) {
        const int rank = s_pre[bin] + mine[bin] + __popc(peers & below);
        if (a.capacity <= 0 || rank < a.capacity) row = s_base[bin] + rank;
        if (row >= a.cap_rows) {  // the row buffer is full: drop the slot and report it
          row = -1;
          if (a.overflow) atomicAdd(a.overflow, 1);
        }
      }
      __syncwarp();
      if (bin >= 0 && (peers & below) == 0u) mine[bin] += __popc(peers);
      __syncwarp();
      if (i < warp_slots && slot < a.n_slots) {
        a.slot_row[slot] = row;
        if (row >= 0) a.row_slot[row] = static_cast<int>(slot);
      }
    }
  }
  // the experts by descending rows, equal ones in order
  if (a.group_order != nullptr) {
    for (int e = unit * T + tid; e < a.n_local; e += gridDim.x * T) {
      const int rows = s_goff[e + 1] - s_goff[e];
      int rank = 0;
      for (int o = 0; o < a.n_local; ++o) {
        const int r = s_goff[o + 1] - s_goff[o];
        rank += r > rows || (r == rows && o < e) ? 1 : 0;
      }
      a.group_order[rank] = e;
    }
  }
  // expert of every tile, spread over the CTAs
  const int tiles = s_goff[a.n_local] / 128, all_tiles = static_cast<int>((a.cap_rows + 127) / 128);
  for (int t = unit * T + tid; t < all_tiles; t += gridDim.x * T) {
    int e = -1;
    if (t < tiles) {
      int lo = 0, hi = a.n_local;  // largest e with goff[e] <= row
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_goff[mid] <= t * 128) lo = mid; else hi = mid;
      }
      e = lo;
      if (a.tile_rows != nullptr) {
        // the rows of an expert are its kept slots, in front of its padding
        int rows = 0;
        for (int k = 0; k < kb; ++k) rows += s_tot[e * kb + k];
        a.tile_rows[t] = max(0, min(128, s_goff[e] + rows - t * 128));
      }
      if (a.pair_tile != nullptr) {
        const int in_group = t - s_goff[e] / 128;
        if ((in_group & 1) == 0) a.pair_tile[s_pair[e] + in_group / 2] = 2 * t + (s_goff[e + 1] <= (t + 1) * 128 ? 1 : 0);
      }
    }
    a.tile_group[t] = e;
  }
}

// Few slots, many bins: one CTA.  The slots are counted by all threads and ranked by one warp, 32 at a time; `work` holds
// the next row and the end of every bin ([2][nbins], shared memory where it fits).
__global__ void __launch_bounds__(1024) plan_sparse_kernel(const MoePlanArgs a, int nbins, int* work) {
  chain_wait();
  chain_trigger();
  extern __shared__ int plan_smem[];
  __shared__ long long s_sum[32];
  int* next = work != nullptr ? work : plan_smem;
  int* end = next + nbins;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int kb = a.per_k_bins ? a.K : 1;
  const int cap128 = static_cast<int>(a.cap_rows / 128 * 128);
  // exclusive prefix over the threads and the total of all of them
  auto block_prefix = [&](long long v, long long& total) {
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    long long before = 0;
    total = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += s_sum[w];
      total += s_sum[w];
    }
    __syncthreads();
    return before + incl - v;
  };

  for (int b = tid; b < nbins; b += 1024) next[b] = 0;
  for (long long r = tid; r < a.cap_rows; r += 1024) a.row_slot[r] = -1;
  __syncthreads();
  for (long long s = tid; s < a.n_slots; s += 1024) {
    const int bin = plan_bin(a, s);
    if (bin >= 0) atomicAdd(next + bin, 1);
  }
  __syncthreads();
  // every thread takes a run of neighbouring experts: their padded rows, the rows before them, then bin by bin
  const int per = (a.n_local + 1023) / 1024;
  const int e0 = min(a.n_local, tid * per), e1 = min(a.n_local, e0 + per);
  auto kept_of = [&](int bin) { return a.capacity > 0 ? min(next[bin], a.capacity) : next[bin]; };
  long long mine = 0, total = 0;
  for (int e = e0; e < e1; ++e) {
    int cnt = 0;
    for (int k = 0; k < kb; ++k) cnt += kept_of(e * kb + k);
    mine += (cnt + 127) / 128 * 128;
  }
  long long raw = block_prefix(mine, total);
  for (int e = e0; e < e1; ++e) {
    const int off = raw < cap128 ? static_cast<int>(raw) : cap128;
    int cnt = 0;
    for (int k = 0; k < kb; ++k) {
      const int bin = e * kb + k, n = kept_of(bin);
      next[bin] = off + cnt;
      cnt += n;
      end[bin] = off + cnt;
    }
    // rows that do not fit the buffer are dropped below (and counted in `overflow`)
    const long long room = a.cap_rows - off;
    a.counts_kept[e] = cnt > room ? static_cast<int>(room > 0 ? room : 0) : cnt;
    a.group_offsets[e] = off;
    raw += (cnt + 127) / 128 * 128;
  }
  if (tid == 0) {
    const int off = total < cap128 ? static_cast<int>(total) : cap128;
    a.group_offsets[a.n_local] = off;
    *a.num_m_tiles = off / 128;
  }
  __syncthreads();
  if (warp == 0) {
    for (long long s0 = 0; s0 < a.n_slots; s0 += 32) {
      const long long slot = s0 + lane;
      const int bin = slot < a.n_slots ? plan_bin(a, slot) : -1;
      const unsigned peers = __match_any_sync(0xffffffffu, bin);
      int row = -1;
      if (bin >= 0) {
        row = next[bin] + __popc(peers & below);
        if (row >= end[bin]) {
          row = -1;  // beyond the capacity
        } else if (row >= a.cap_rows) {  // the row buffer is full: drop the slot and report it
          row = -1;
          if (a.overflow) atomicAdd(a.overflow, 1);
        }
      }
      __syncwarp();
      if (bin >= 0 && (peers & below) == 0u) next[bin] += __popc(peers);
      __syncwarp();
      if (slot < a.n_slots) {
        a.slot_row[slot] = row;
        if (row >= 0) a.row_slot[row] = static_cast<int>(slot);
      }
    }
  }
  __syncthreads();
  if (a.pair_tile != nullptr) {  // the first pair of every expert, where the bins were
    long long n = 0;
    for (int e = e0; e < e1; ++e) n += (a.group_offsets[e + 1] - a.group_offsets[e] + 255) / 256;
    long long first = block_prefix(n, total);
    for (int e = e0; e < e1; ++e) {
      next[e] = static_cast<int>(first);
      first += (a.group_offsets[e + 1] - a.group_offsets[e] + 255) / 256;
    }
    if (tid == 0) *a.num_pairs = static_cast<int>(total);
    __syncthreads();
  }
  const int* goff = a.group_offsets;
  if (a.group_order != nullptr) {
    for (int e = tid; e < a.n_local; e += 1024) {
      const int rows = goff[e + 1] - goff[e];
      int rank = 0;
      for (int o = 0; o < a.n_local; ++o) {
        const int r = goff[o + 1] - goff[o];
        rank += r > rows || (r == rows && o < e) ? 1 : 0;
      }
      a.group_order[rank] = e;
    }
  }
  const int tiles = goff[a.n_local] / 128, all_tiles = static_cast<int>((a.cap_rows + 127) / 128);
  for (int t = tid; t < all_tiles; t += 1024) {
    int e = -1;
    if (t < tiles) {
      int lo = 0, hi = a.n_local;  // largest e with goff[e] <= row
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (goff[mid] <= t * 128) lo = mid; else hi = mid;
      }
      e = lo;
      if (a.tile_rows != nullptr) a.tile_rows[t] = max(0, min(128, goff[e] + a.counts_kept[e] - t * 128));
      if (a.pair_tile != nullptr) {
        const int in_group = t - goff[e] / 128;
        if ((in_group & 1) == 0) a.pair_tile[next[e] + in_group / 2] = 2 * t + (goff[e + 1] <= (t + 1) * 128 ? 1 : 0);
      }
    }
    a.tile_group[t] = e;
  }
}

struct PlanShape {
  int nbins, unit_slots, n_units;
  bool single, scan, wide;  // wide: the ranking kernel's working storage lies in global memory
  bool sparse;              // few slots over bins that do not fit the ranking kernel's shared memory
  PlanShape(long long n_slots, int n_local, int K, int per_k_bins) {
    nbins = n_local * (per_k_bins ? K : 1);
    single = n_slots <= kSingleSlots && rank_words(kWarpsSingle, nbins, n_local) * 4 <= kSmemLimit;
    wide = !single && rank_words(kWarpsMulti, nbins, n_local) * 4 > kSmemLimit;
    sparse = wide && n_slots <= kSparseSlots;
    // a unit has at least as many slots as bins twice over, so that its histogram is not larger than its slots
    unit_slots = single ? static_cast<int>((n_slots + 1023) / 1024 * 1024) : 1024 * ((nbins + 511) / 512);
    n_units = single ? 1 : static_cast<int>((n_slots + unit_slots - 1) / unit_slots);
    scan = !single && static_cast<long long>(n_units) * nbins > kRedundantWords;
  }
  bool sparse_in_smem() const { return 8ll * nbins <= kSmemLimit; }
  long long hist_words() const { return single ? 0 : (static_cast<long long>(n_units) + 1) * nbins; }
};

}  // namespace

size_t moe_plan_scratch_words(long long n_slots, int n_local, int K, int per_k_bins) {
  const PlanShape s(n_slots, n_local, K, per_k_bins);
  if (s.sparse) return s.sparse_in_smem() ? 1 : 2 * static_cast<size_t>(s.nbins);
  const long long work = s.wide ? s.n_units * rank_words(kWarpsMulti, s.nbins, n_local) : 0;
  return static_cast<size_t>(s.hist_words() + work + 1);
}

// Launches with more than the 48 KiB of shared memory that need no asking for.  Asked for on every such call: the answer
// belongs to one device, and a process may plan on several.
template <typename... P, typename... A>
static cudaError_t launch_large(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                                A&&... args) {
  if (smem > 47 * 1024) {  // the rest is for the kernels' fixed arrays
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(kernel, grid, threads, smem, stream, std::forward<A>(args)...);
}

cudaError_t launch_moe_plan(const MoePlanArgs& a, cudaStream_t stream) {
  if (a.n_slots <= 0 || a.n_local <= 0) return cudaErrorInvalidValue;
  const PlanShape s(a.n_slots, a.n_local, a.K, a.per_k_bins);
  if (s.single) {
    const size_t smem = rank_words(kWarpsSingle, s.nbins, a.n_local) * 4;
    return launch_large(plan_rank_kernel<kWarpsSingle, true>, 1, kWarpsSingle * 32, smem, stream, a, s.nbins,
                          s.unit_slots, 1, 0, nullptr);
  }
  if (s.sparse) {
    const bool in_smem = s.sparse_in_smem();
    return launch_large(plan_sparse_kernel, 1, 1024, in_smem ? 8ull * s.nbins : 0, stream, a, s.nbins,
                          in_smem ? nullptr : a.scratch);
  }
  const bool hist_in_smem = s.nbins * 4 <= 48 * 1024;
  cudaError_t e = launch_chained(plan_count_kernel, s.n_units, kCountThreads, hist_in_smem ? s.nbins * 4 : 0, stream, a,
                                 s.nbins, s.unit_slots, hist_in_smem ? 1 : 0);
  if (e != cudaSuccess) return e;
  if (s.scan) e = launch_chained(plan_scan_kernel, (s.nbins + 31) / 32, 1024, 0, stream, a, s.nbins, s.n_units);
  if (e != cudaSuccess) return e;
  const size_t smem = s.wide ? 0 : rank_words(kWarpsMulti, s.nbins, a.n_local) * 4;
  return launch_large(plan_rank_kernel<kWarpsMulti, false>, s.n_units, kWarpsMulti * 32, smem, stream, a, s.nbins,
                        s.unit_slots, s.n_units, s.scan ? 1 : 0, s.wide ? a.scratch + s.hist_words() : nullptr);
}

}  // namespace cmoe
