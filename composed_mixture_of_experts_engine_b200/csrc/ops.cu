// Bandwidth-bound kernels of the training step: RMSNorm, RoPE, fused AdamW (+ global-norm clipping
// without a host round trip), cross-entropy with in-place gradient, and the MoE row kernels (row gather, weighted
// combine; the row plan is in plan.cu).
//
// Reference counterparts: RMSNorm eager ops (pkg/models/moe.py:83-86); torch.optim.AdamW +
// clip_grad_norm_ + F.cross_entropy (train.py:207-212, 297-303, 322-323); the per-k scatter loop of the
// MoE layer (pkg/distributed/moe_layer.py:309-353).  RoPE has no counterpart there.
#include "ops.cuh"

#include <climits>
#include <cstdlib>

#include "common.cuh"
#include "launch.h"

namespace cmoe {

namespace {

__device__ __forceinline__ void unpack8(const uint4& x, float (&f)[8]) {
  const float2 a = unpack_bf16x2(x.x), b = unpack_bf16x2(x.y), c = unpack_bf16x2(x.z), d = unpack_bf16x2(x.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  unpack8(*reinterpret_cast<const uint4*>(p), f);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 o;
  o.x = pack_bf16x2(f[0], f[1]);
  o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]);
  o.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = o;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (threadIdx.x < THREADS / 32) ? red[threadIdx.x] : 0.f;
  if (warp == 0) {
    t = warp_sum(t);
    if (lane == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}

// ------------------------------------------------------------------------------------ RMSNorm
// One CTA of 128 threads per row; each thread keeps VEC vectors of 8 columns in registers
// (VEC = 1, 2, 4, 8 covers H <= 1024, 2048, 4096, 8192).  Small CTAs keep 16 rows in flight per SM.
constexpr int RN_THREADS = 128;

// ADD: the row is x + delta, rounded to bf16 and written to `sum` first (a residual stream and the branch that joins it:
// one pass instead of an addition of its own and a pass that reads its result).
template <int VEC, bool ADD>
__global__ void __launch_bounds__(RN_THREADS) rmsnorm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* delta,
                                                                 __nv_bfloat16* sum, const __nv_bfloat16* w,
                                                                 __nv_bfloat16* y,
                                                                 float* rstd, long long rows, int H,
                                                                 float eps) {
  chain_wait();
  chain_trigger();
  __shared__ float red[RN_THREADS / 32];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16* xr = x + row * H;
    float v[VEC][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * RN_THREADS + threadIdx.x) * 8;
      if (c < H) {
        load8(xr + c, v[i]);
        if (ADD) {
          float d[8];
          load8(delta + row * H + c, d);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = __bfloat162float(__float2bfloat16(v[i][j] + d[j]));
          store8(sum + row * H + c, v[i]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += v[i][j] * v[i][j];
      }
    }
    ss = block_sum<RN_THREADS>(ss, red);
    const float r = rsqrtf(ss / H + eps);
    if (threadIdx.x == 0 && rstd) rstd[row] = r;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * RN_THREADS + threadIdx.x) * 8;
      if (c < H) {
        float wv[8], o[8];
        load8(w + c, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = v[i][j] * r * wv[j];
        store8(y + row * H + c, o);
      }
    }
  }
}

// rows of x / dy that a CTA of the backward kernel keeps in flight (shared-memory ring)
__host__ __device__ constexpr int rn_bwd_stages(int vec) { return vec <= 2 ? 4 : 2; }
__host__ __device__ constexpr int rn_bwd_smem(int vec, int streams) { return rn_bwd_stages(vec) * streams * vec * RN_THREADS * 16; }

__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
               "l"(gsrc)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// RES: `dres`, the gradient that reaches the row past the norm (a residual stream), is added to dx before it is rounded.
template <int VEC, bool RES>
__global__ void __launch_bounds__(RN_THREADS) rmsnorm_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* dres,
                                                                 const __nv_bfloat16* x,
                                                                 const __nv_bfloat16* w,
                                                                 const float* rstd,
                                                                 __nv_bfloat16* dx, float* dw,
                                                                 float* dw_partial, long long rows,
                                                                 int H) {
  chain_wait();
  chain_trigger();
  __shared__ float red[RN_THREADS / 32];
  extern __shared__ uint4 rn_ring[];  // [stages][x | dy | dres][VEC][RN_THREADS]: every thread's own 16-byte pieces
  constexpr int S = rn_bwd_stages(VEC), STREAMS = RES ? 3 : 2;
  float wv[VEC][8], dwacc[VEC][8];
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    const int c = (i * RN_THREADS + threadIdx.x) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dwacc[i][j] = 0.f;
      wv[i][j] = 0.f;
    }
    if (c < H) load8(w + c, wv[i]);
  }
  // The rows of x and dy stream through a ring of S rows in shared memory, filled by per-thread asynchronous copies
  // (`cp.async`, 16 bytes each, past L1): a CTA keeps S rows of loads in flight without holding them in registers,
  // and every thread reads back only the pieces it copied itself, so the ring needs no barrier.  One commit group per
  // row (an empty one past the end), so that "all but the newest S - 1 groups" is always the row about to be used.
  auto slot = [&](int s, int which, int i) { return rn_ring + ((s * STREAMS + which) * VEC + i) * RN_THREADS + threadIdx.x; };
  auto issue = [&](long long row, int s) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * RN_THREADS + threadIdx.x) * 8;
      if (row < rows && c < H) {
        cp_async_16(slot(s, 0, i), x + row * H + c);
        cp_async_16(slot(s, 1, i), dy + row * H + c);
        if (RES) cp_async_16(slot(s, 2, i), dres + row * H + c);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < S; ++s) issue(blockIdx.x + static_cast<long long>(s) * gridDim.x, s);
  int s = 0;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    cp_async_wait<S - 1>();
    const float r = rstd[row];
    float xh[VEC][8], g[VEC][8];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * RN_THREADS + threadIdx.x) * 8;
      if (c < H) {
        const uint4 nx = *slot(s, 0, i), nd = *slot(s, 1, i);
        const uint32_t xw[4] = {nx.x, nx.y, nx.z, nx.w};
        const uint32_t dw4[4] = {nd.x, nd.y, nd.z, nd.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 xv = unpack_bf16x2(xw[q]), dv = unpack_bf16x2(dw4[q]);
          xh[i][2 * q] = xv.x * r;
          xh[i][2 * q + 1] = xv.y * r;
          g[i][2 * q] = dv.x * wv[i][2 * q];
          g[i][2 * q + 1] = dv.y * wv[i][2 * q + 1];
          dot += g[i][2 * q] * xh[i][2 * q] + g[i][2 * q + 1] * xh[i][2 * q + 1];
          dwacc[i][2 * q] += dv.x * xh[i][2 * q];
          dwacc[i][2 * q + 1] += dv.y * xh[i][2 * q + 1];
        }
        if (RES) {  // g becomes what of dx does not wait for the row's sum
          float f[8];
          unpack8(*slot(s, 2, i), f);
#pragma unroll
          for (int j = 0; j < 8; ++j) g[i][j] = fmaf(r, g[i][j], f[j]);
        }
      }
    }
    // Refill the slot with the row S steps ahead.  Its three pieces were read by this thread, which alone writes them, before
    // this line: the copy's asm statement lets no read of memory past it, and a thread's own reads are ahead of a copy that
    // it starts later.  (The sums above have used all of them, so no raw piece is held across the copy.)
    issue(row + static_cast<long long>(S) * gridDim.x, s);
    s = (s + 1 == S) ? 0 : s + 1;
    dot = block_sum<RN_THREADS>(dot, red) / H;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * RN_THREADS + threadIdx.x) * 8;
      if (c < H) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = RES ? g[i][j] - xh[i][j] * (r * dot) : r * (g[i][j] - xh[i][j] * dot);
        store8(dx + row * H + c, o);
      }
    }
  }
  if (dw_partial) {
    // one row of partial column sums per CTA, summed in a fixed order by the colsum kernels: CTAs adding atomically to
    // the same H addresses serialise in L2 and cost more than the whole row pass
    float* out = dw_partial + static_cast<long long>(blockIdx.x) * H;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * RN_THREADS + threadIdx.x) * 8;
      if (c < H) {
        *reinterpret_cast<float4*>(out + c) = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
        *reinterpret_cast<float4*>(out + c + 4) = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
      }
    }
  } else if (dw) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * RN_THREADS + threadIdx.x) * 8;
      if (c < H) {
#pragma unroll
        for (int j = 0; j < 8; ++j) atomicAdd(dw + c + j, dwacc[i][j]);
      }
    }
  }
}

// dw[c] += column sums of the per-CTA partial rows, in a fixed order (the same inputs give the same bits, whichever CTA
// finishes first): 16 warps take every 16th row each, a lane per column, and their sums are added in order.  What bounds
// it: latency.  In two launches (slices of rows, then the slices' sums) it took 13.4 us for 592 rows of 1024.
constexpr int CSUM_WARPS = 16;
__global__ void __launch_bounds__(CSUM_WARPS * 32) colsum_kernel(const float* partial, float* dw, int n_rows, int H) {
  chain_wait();
  chain_trigger();
  __shared__ float sums[CSUM_WARPS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < H)
#pragma unroll 8
    for (int b = warp; b < n_rows; b += CSUM_WARPS) s += partial[static_cast<long long>(b) * H + c];  // loads ahead, adds in order
  sums[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || c >= H) return;
#pragma unroll
  for (int w = 1; w < CSUM_WARPS; ++w) s += sums[w][lane];
  dw[c] += s;
}

// ------------------------------------------------------------------------------------ RoPE
__global__ void rope_kernel(__nv_bfloat16* t, const float* cos_tab,
                            const float* sin_tab, long long rows, int seq, int heads, int head_dim,
                            long long row_stride, int inverse) {
  chain_wait();
  chain_trigger();
  const int half = head_dim / 2;
  const int vec_per_head = half / 8;
  const long long total = rows * heads * vec_per_head;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int vi = static_cast<int>(i % vec_per_head);
    const long long rh = i / vec_per_head;
    const int h = static_cast<int>(rh % heads);
    const long long r = rh / heads;
    const int pos = static_cast<int>(r % seq);
    __nv_bfloat16* base = t + r * row_stride + static_cast<long long>(h) * head_dim + vi * 8;
    float a[8], b[8], oa[8], ob[8];
    load8(base, a);
    load8(base + half, b);
    const float* cp = cos_tab + static_cast<long long>(pos) * half + vi * 8;
    const float* sp = sin_tab + static_cast<long long>(pos) * half + vi * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float c = cp[j];
      const float s = inverse ? -sp[j] : sp[j];
      oa[j] = a[j] * c - b[j] * s;
      ob[j] = b[j] * c + a[j] * s;
    }
    store8(base, oa);
    store8(base + half, ob);
  }
}

// Packs the three attention gradients into one [rows, heads, head_dim] buffer (q heads, k heads, v heads) and undoes
// the rotary embedding on the q and k heads on the way: one read and one write of every element instead of three
// strided copies plus an in-place rotation pass.  Sources are [B, h, S, head_dim] views with arbitrary batch / head /
// sequence strides and unit stride on head_dim.
struct QkvGradSrc {
  const __nv_bfloat16* ptr;
  long long sb, sh, ss;  // strides (elements) of batch, head, sequence position
};

__global__ void qkv_grad_pack_kernel(QkvGradSrc dq, QkvGradSrc dk, QkvGradSrc dv, __nv_bfloat16* out,
                                     const float* cos_tab, const float* sin_tab,
                                     long long rows, int seq, int nh, int nkv, int head_dim) {
  chain_wait();
  chain_trigger();
  const int heads = nh + 2 * nkv;
  const int half = head_dim / 2;
  const int vec_per_head = half / 8;
  const long long total = rows * heads * vec_per_head;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int vi = static_cast<int>(i % vec_per_head);
    const long long rh = i / vec_per_head;
    const int h = static_cast<int>(rh % heads);
    const long long r = rh / heads;
    const int pos = static_cast<int>(r % seq);
    const long long b = r / seq;
    const QkvGradSrc& s = h < nh ? dq : (h < nh + nkv ? dk : dv);
    const int hh = h < nh ? h : (h < nh + nkv ? h - nh : h - nh - nkv);
    const __nv_bfloat16* src = s.ptr + b * s.sb + hh * s.sh + pos * s.ss + vi * 8;
    __nv_bfloat16* dst = out + (r * heads + h) * head_dim + vi * 8;
    const uint4 ra = __ldcs(reinterpret_cast<const uint4*>(src));
    const uint4 rb = __ldcs(reinterpret_cast<const uint4*>(src + half));
    if (h >= nh + nkv) {  // v heads: plain copy
      *reinterpret_cast<uint4*>(dst) = ra;
      *reinterpret_cast<uint4*>(dst + half) = rb;
      continue;
    }
    const uint32_t aw[4] = {ra.x, ra.y, ra.z, ra.w}, bw[4] = {rb.x, rb.y, rb.z, rb.w};
    uint32_t oa[4], ob[4];
    const float* cp = cos_tab + static_cast<long long>(pos) * half + vi * 8;
    const float* sp = sin_tab + static_cast<long long>(pos) * half + vi * 8;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 a = unpack_bf16x2(aw[q]), bb = unpack_bf16x2(bw[q]);
      const float c0 = cp[2 * q], c1 = cp[2 * q + 1], s0 = sp[2 * q], s1 = sp[2 * q + 1];
      // the transpose of the rotation: [a; b] -> [a c + b s; b c - a s]
      oa[q] = pack_bf16x2(a.x * c0 + bb.x * s0, a.y * c1 + bb.y * s1);
      ob[q] = pack_bf16x2(bb.x * c0 - a.x * s0, bb.y * c1 - a.y * s1);
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(oa[0], oa[1], oa[2], oa[3]);
    *reinterpret_cast<uint4*>(dst + half) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
  }
}

// ------------------------------------------------------------------------------------ AdamW
struct AdamWCoeffs {
  float gs, inv_bc1, inv_sqrt_bc2, decay, omb1, omb2;
};
__device__ __forceinline__ AdamWCoeffs adamw_coeffs(const AdamWArgs& a) {
  AdamWCoeffs c;
  c.gs = a.grad_scale;
  if (a.max_norm > 0.f && a.sumsq != nullptr) {
    const float norm = sqrtf(*a.sumsq);  // sumsq already refers to the scaled gradients
    c.gs *= fminf(1.f, a.max_norm / (norm + 1e-6f));
  }
  c.inv_bc1 = 1.f / a.bias_corr1;
  c.inv_sqrt_bc2 = rsqrtf(a.bias_corr2);
  c.decay = 1.f - a.lr * a.weight_decay;
  c.omb1 = 1.f - a.beta1;
  c.omb2 = 1.f - a.beta2;
  return c;
}
__device__ __forceinline__ void adamw_update(const AdamWArgs& a, const AdamWCoeffs& c, float g, float& p, float& m, float& v) {
  const float gj = g * c.gs;
  m = a.beta1 * m + c.omb1 * gj;
  v = a.beta2 * v + c.omb2 * gj * gj;
  const float denom = sqrtf(v) * c.inv_sqrt_bc2 + a.eps;
  p = p * c.decay - a.lr * (m * c.inv_bc1) * __frcp_rn(denom);
}

// fp32 gradients, n a multiple of 8, pointers on 32-byte boundaries: eight elements per thread in 32-byte accesses, a thread
// per eight elements.  What bounds it: 34 bytes of memory traffic per parameter.  A grid that strides over the buffers with
// 16-byte accesses (the form below) left a quarter of the rate unused, its threads wait for their loads with every step:
// 400 M parameters behind GEMMs 2474 / 1996 us (6.8 TB/s), 100 M 631 / 513, 8 M 52 / 49, 1 M 15.3 / 13.3.  Of the
// difference the one-shot grid is the larger part (16-byte accesses in it: 2170), streaming hints on the stores cost (2177
// with, 2027 without, two 16-byte pieces per thread).
__device__ __forceinline__ void load32(const float* p, float (&r)[8]) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void store32(float* p, const float (&r)[8]) {
  asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]),
               "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "l"(p)
               : "memory");
}
__global__ void __launch_bounds__(256) adamw_wide_kernel(const AdamWArgs a) {
  chain_wait();
  chain_trigger();
  const long long i = (blockIdx.x * 256LL + threadIdx.x) * 8;
  if (i >= a.n) return;
  float* grad = static_cast<float*>(const_cast<void*>(a.grad));
  float p[8], m[8], v[8], g[8];
  load32(a.p32 + i, p);
  load32(a.m + i, m);
  load32(a.v + i, v);
  load32(grad + i, g);
  const AdamWCoeffs c = adamw_coeffs(a);
#pragma unroll
  for (int j = 0; j < 8; ++j) adamw_update(a, c, g[j], p[j], m[j], v[j]);
  store32(a.p32 + i, p);
  store32(a.m + i, m);
  store32(a.v + i, v);
  if (a.p16) store8(static_cast<__nv_bfloat16*>(a.p16) + i, p);
  if (a.zero_grad) {
    const float zero[8] = {};
    store32(grad + i, zero);
  }
}

// any other form
__global__ void adamw_kernel(const AdamWArgs a) {
  chain_wait();
  chain_trigger();
  const AdamWCoeffs c = adamw_coeffs(a);
  const float gs = c.gs, inv_bc1 = c.inv_bc1, inv_sqrt_bc2 = c.inv_sqrt_bc2;
  const long long n4 = a.n / 4;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  float4* __restrict__ p32v = reinterpret_cast<float4*>(a.p32);
  float4* __restrict__ mv = reinterpret_cast<float4*>(a.m);
  float4* __restrict__ vv4 = reinterpret_cast<float4*>(a.v);
  uint2* __restrict__ p16v = reinterpret_cast<uint2*>(a.p16);
  float4* __restrict__ g32v = reinterpret_cast<float4*>(const_cast<void*>(a.grad));
  uint2* __restrict__ g16v = reinterpret_cast<uint2*>(const_cast<void*>(a.grad));
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4; i += stride) {
    // all loads first (streaming: nothing here is read twice), then the math, then the stores
    const float4 p = __ldcs(p32v + i);
    const float4 m = __ldcs(mv + i);
    const float4 v = __ldcs(vv4 + i);
    float g[4];
    if (a.grad_is_bf16) {
      const uint2 raw = __ldcs(g16v + i);
      const float2 g0 = unpack_bf16x2(raw.x), g1 = unpack_bf16x2(raw.y);
      g[0] = g0.x; g[1] = g0.y; g[2] = g1.x; g[3] = g1.y;
    } else {
      const float4 raw = __ldcs(g32v + i);
      g[0] = raw.x; g[1] = raw.y; g[2] = raw.z; g[3] = raw.w;
    }
    float pp[4] = {p.x, p.y, p.z, p.w}, mm[4] = {m.x, m.y, m.z, m.w}, vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) adamw_update(a, c, g[j], pp[j], mm[j], vv[j]);
    __stcs(p32v + i, make_float4(pp[0], pp[1], pp[2], pp[3]));
    __stcs(mv + i, make_float4(mm[0], mm[1], mm[2], mm[3]));
    __stcs(vv4 + i, make_float4(vv[0], vv[1], vv[2], vv[3]));
    if (a.p16) p16v[i] = make_uint2(pack_bf16x2(pp[0], pp[1]), pack_bf16x2(pp[2], pp[3]));
    if (a.zero_grad) {
      if (a.grad_is_bf16) __stcs(g16v + i, make_uint2(0u, 0u));
      else __stcs(g32v + i, make_float4(0.f, 0.f, 0.f, 0.f));
    }
  }
  // tail (n not a multiple of 4)
  const long long tail0 = n4 * 4;
  const long long gi = tail0 + blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (gi < a.n) {
    float g = a.grad_is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.grad)[gi])
                             : reinterpret_cast<const float*>(a.grad)[gi];
    if (a.zero_grad) {
      if (a.grad_is_bf16) reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(a.grad))[gi] = __float2bfloat16(0.f);
      else reinterpret_cast<float*>(const_cast<void*>(a.grad))[gi] = 0.f;
    }
    g *= gs;
    const float m = a.beta1 * a.m[gi] + (1.f - a.beta1) * g;
    const float v = a.beta2 * a.v[gi] + (1.f - a.beta2) * g * g;
    const float denom = sqrtf(v) * inv_sqrt_bc2 + a.eps;
    const float p = a.p32[gi] * (1.f - a.lr * a.weight_decay) - a.lr * (m * inv_bc1) / denom;
    a.p32[gi] = p;
    a.m[gi] = m;
    a.v[gi] = v;
    if (a.p16) reinterpret_cast<__nv_bfloat16*>(a.p16)[gi] = __float2bfloat16(p);
  }
}

__global__ void __launch_bounds__(256) sumsq_kernel(const void* x, int is_bf16, long long n, float* out,
                                                    float* partials) {
  chain_wait();
  chain_trigger();
  __shared__ float red[8];
  float acc = 0.f;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  if (is_bf16) {
    const long long n8 = n / 8;
    const __nv_bfloat16* xb = reinterpret_cast<const __nv_bfloat16*>(x);
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n8; i += stride) {
      float f[8];
      load8(xb + i * 8, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc += f[j] * f[j];
    }
    const long long gi = n8 * 8 + blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (gi < n) {
      const float f = __bfloat162float(xb[gi]);
      acc += f * f;
    }
  } else {
    const long long n4 = n / 4;
    const float* xf = reinterpret_cast<const float*>(x);
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4; i += stride) {
      const float4 f = reinterpret_cast<const float4*>(xf)[i];
      acc += f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w;
    }
    const long long gi = n4 * 4 + blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (gi < n) acc += xf[gi] * xf[gi];
  }
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) {
    if (partials != nullptr)
      partials[blockIdx.x] = acc;  // summed in block order by sumsq_final_kernel
    else
      atomicAdd(out, acc);
  }
}

// out += sum of `n` per-block partial sums, always in the same order (one block, fixed tree)
__global__ void __launch_bounds__(256) sumsq_final_kernel(const float* partials, int n,
                                                          float* out) {
  chain_wait();
  chain_trigger();
  __shared__ float red[8];
  float acc = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) acc += partials[i];
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) *out += acc;
}

// Sum of the partial results of a contraction that was cut into `parts` pieces, always in the same order; the result
// replaces or is added to fp32, or is rounded once to bf16.
template <int OUT>  // 0: fp32 store, 1: fp32 add, 2: bf16 store
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float4* part, int parts, long long n4,
                                                            void* out) {
  chain_wait();
  chain_trigger();
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= n4) return;
  float4 acc = __ldcs(part + i);
#pragma unroll 8
  for (int s = 1; s < parts; ++s) {
    const float4 v = __ldcs(part + s * n4 + i);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  if (OUT == 2) {
    reinterpret_cast<uint2*>(out)[i] = make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
  } else {
    float4* o = reinterpret_cast<float4*>(out) + i;
    if (OUT == 1) {
      const float4 v = *o;
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    *o = acc;
  }
}

// ------------------------------------------------------------------------------------ cross-entropy
constexpr int CE_THREADS = 512;
__global__ void __launch_bounds__(CE_THREADS) cross_entropy_kernel(__nv_bfloat16* logits,
                                                                   const long long* targets,
                                                                   float* loss_sum,
                                                                   float* row_loss, long long rows, int V,
                                                                   long long ld, float grad_scale) {
  chain_wait();
  chain_trigger();
  __shared__ float red[CE_THREADS / 32];
  __shared__ float s_max, s_sum;
  const long long row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const long long tgt = targets[row];
  const int nvec = V / 8;
  // online max / sum-exp per thread, then merged across the block
  float mx = -INFINITY, se = 0.f;
  for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
    float f[8];
    load8(lr + i * 8, f);
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    if (lm > mx) {
      se *= __expf(mx - lm);
      mx = lm;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) se += __expf(f[j] - mx);
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += CE_THREADS) {
    const float f = __bfloat162float(lr[c]);
    if (f > mx) {
      se *= __expf(mx - f);
      mx = f;
    }
    se += __expf(f - mx);
  }
  // block max
  float bm = warp_max(mx);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = bm;
  __syncthreads();
  if (warp == 0) {
    float t = lane < CE_THREADS / 32 ? red[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) s_max = t;
  }
  __syncthreads();
  bm = s_max;
  se = (mx == -INFINITY) ? 0.f : se * __expf(mx - bm);
  se = block_sum<CE_THREADS>(se, red);
  if (threadIdx.x == 0) s_sum = se;
  __syncthreads();
  const float lse = bm + logf(s_sum);
  const bool ignore = tgt < 0 || tgt >= V;
  if (threadIdx.x == 0) {
    const float l = ignore ? 0.f : lse - __bfloat162float(lr[tgt]);
    if (row_loss != nullptr)
      row_loss[row] = l;  // the caller sums the rows in a fixed order
    else if (!ignore)
      atomicAdd(loss_sum, l);
  }
  __syncthreads();
  const float gs = ignore ? 0.f : grad_scale;
  for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
    float f[8], o[8];
    load8(lr + i * 8, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float p = __expf(f[j] - lse);
      o[j] = (p - ((i * 8 + j) == tgt ? 1.f : 0.f)) * gs;
    }
    store8(lr + i * 8, o);
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += CE_THREADS) {
    const float p = __expf(__bfloat162float(lr[c]) - lse);
    lr[c] = __float2bfloat16((p - (c == tgt ? 1.f : 0.f)) * gs);
  }
}

// The same loss and gradient where the GEMM that made the logits has left the maximum and the sum of exp(v - maximum) of
// every 256 columns (GemmArgs::row_stats): the row is read and written once, with one exponential per logit.  What bounds
// it: these passes, which take as long as a copy.  4096 x 50304 behind GEMMs, at the clock that these leave: 279 us with
// the row read twice, 147 this way (a copy: 138); 4096 x 8192 77 / 36.  Small CTAs, whose first loads are in flight while
// the statistics are merged, measured better than large ones: 256 threads 147, 512 155, 1024 177.
constexpr int CS_THREADS = 256, CS_VECS = 2;
__global__ void __launch_bounds__(CS_THREADS) cross_entropy_stats_kernel(__nv_bfloat16* logits, const float2* stats,
                                                                         const long long* targets, float* loss_sum,
                                                                         float* row_loss, int V, long long ld,
                                                                         float grad_scale) {
  chain_wait();
  chain_trigger();
  __shared__ float warp_m[CS_THREADS / 32], warp_s[CS_THREADS / 32];
  const long long row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const long long tgt = targets[row];
  const int nvec = V / 8;  // V is a multiple of 8
  uint4 v[CS_VECS];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int q = 0; q < CS_VECS; ++q)
      if (i0 + q * CS_THREADS < nvec) v[q] = reinterpret_cast<const uint4*>(lr)[i0 + q * CS_THREADS];
  };
  fetch(threadIdx.x);
  const int n = (V + 255) / 256;
  float mx = -INFINITY, se = 0.f;
  // sums of parts without a finite or larger value are 0 and stay so
  const auto scaled = [](float s, float m, float to) { return m == -INFINITY ? (isnan(s) ? s : 0.f) : s * __expf(m - to); };
  for (int i = threadIdx.x; i < n; i += CS_THREADS) {
    const float2 s = stats[row * n + i];
    const float m = fmaxf(mx, s.x);
    se = scaled(se, mx, m) + scaled(s.y, s.x, m);
    mx = m;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float wm = warp_max(mx), ws = warp_sum(scaled(se, mx, wm));
  if (lane == 0) {
    warp_m[warp] = wm;
    warp_s[warp] = ws;
  }
  __syncthreads();
  const float m = lane < CS_THREADS / 32 ? warp_m[lane] : -INFINITY, s = lane < CS_THREADS / 32 ? warp_s[lane] : 0.f;
  const float bm = warp_max(m), lse = bm + logf(warp_sum(scaled(s, m, bm)));
  const bool ignore = tgt < 0 || tgt >= V;
  if (threadIdx.x == 0) {
    const float l = ignore ? 0.f : lse - __bfloat162float(lr[tgt]);
    if (row_loss != nullptr)
      row_loss[row] = l;
    else if (!ignore)
      atomicAdd(loss_sum, l);
  }
  __syncthreads();  // the target's logit has been read
  const float gs = ignore ? 0.f : grad_scale;
  for (int i0 = threadIdx.x; i0 < nvec; i0 += CS_VECS * CS_THREADS) {
    if (i0 != static_cast<int>(threadIdx.x)) fetch(i0);
#pragma unroll
    for (int q = 0; q < CS_VECS; ++q) {
      const int i = i0 + q * CS_THREADS;
      if (i >= nvec) break;
      float f[8], o[8];
      unpack8(v[q], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = __expf(f[j] - lse) * gs;
      const long long at = tgt - i * 8LL;
      if (at >= 0 && at < 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j == at) o[j] = (__expf(f[j] - lse) - 1.f) * gs;
      }
      store8(lr + i * 8, o);
    }
  }
}

// out (+)= *scale * x in fp32, or out = *scale * x in bf16.  One pass over each; what bounds it is those passes.  Library
// operations took a multiply, a cast and a temporary for the second, and 361 us for 103 M elements of the first.
template <int OUT>  // 0: fp32 store, 1: fp32 add, 2: bf16 store
__global__ void __launch_bounds__(256) scaled_out_kernel(const float4* x, const float* scale,
                                                         long long n4, void* out) {
  chain_wait();
  chain_trigger();
  const float s = *scale;
  const long long i0 = blockIdx.x * 1024ll + threadIdx.x;
  float4 v[4], o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long i = i0 + q * 256;
    if (i < n4) {
      v[q] = __ldcs(x + i);
      if (OUT == 1) o[q] = __ldcs(reinterpret_cast<const float4*>(out) + i);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long i = i0 + q * 256;
    if (i < n4) {
      if (OUT == 1)
        __stcs(reinterpret_cast<float4*>(out) + i, make_float4(o[q].x + s * v[q].x, o[q].y + s * v[q].y,
                                                               o[q].z + s * v[q].z, o[q].w + s * v[q].w));
      else if (OUT == 0)
        reinterpret_cast<float4*>(out)[i] = make_float4(s * v[q].x, s * v[q].y, s * v[q].z, s * v[q].w);
      else
        reinterpret_cast<uint2*>(out)[i] = make_uint2(pack_bf16x2(s * v[q].x, s * v[q].y), pack_bf16x2(s * v[q].z, s * v[q].w));
    }
  }
}

// out = *scale * x for bf16 rows, the scale rounded to bf16 first (the library's product with a bf16 scalar, which took 63 us
// for 20 M elements, a broadcast scalar being outside its vectorised kernels; this takes 14).
__global__ void __launch_bounds__(256) scaled_bf16_kernel(const uint4* x, const float* scale, long long n8, uint4* out) {
  chain_wait();
  chain_trigger();
  const float s = __bfloat162float(__float2bfloat16(*scale));
  const long long i0 = blockIdx.x * 1024ll + threadIdx.x;
  uint4 v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (i0 + q * 256 < n8) v[q] = x[i0 + q * 256];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (i0 + q * 256 >= n8) break;
    float f[8];
    unpack8(v[q], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] *= s;
    store8(reinterpret_cast<__nv_bfloat16*>(out + i0 + q * 256), f);
  }
}

// ------------------------------------------------------------------------------------ embedding gradient
// main[keys[i]] += sum over the run of equal keys of dy[order[j]].  Runs are cut at every kEmbSeg sorted positions, a CTA
// per piece (the CTAs of the other positions leave at once): a piece that is a whole run is added to main directly,
// pieces of a longer run are written to `partial` (two rows of H per kEmbSeg positions: [0] of a run that comes in from
// the left, [1] of one that starts here and goes on) and added up, in order, by the join kernel.  So every row of main
// has one writer and a fixed order of additions, and a token that fills the batch is no longer a chain of dependent reads
// in one CTA.  What bounds it: dy once and the touched rows of main twice (16384 tokens of 2048, all distinct: 67 +
// 268 MB, 51 us at the copy rate).  Both kernels, 16384 x 2048, a CTA per run before / now: all distinct 62 / 71 us, uniform
// over 50304 ids 58 / 79, one id 5954 to 10068 / 85, Zipf 905 / 65, every second id the same 5161 / 66.
constexpr int kEmbSeg = 32;  // one ballot finds a piece's end and its source rows
__global__ void __launch_bounds__(256) embedding_grad_kernel(const __nv_bfloat16* dy,
                                                             const long long* keys,
                                                             const long long* order,
                                                             float* main, float* partial, int n, int H) {
  chain_wait();
  chain_trigger();
  const int i = blockIdx.x;
  const int lane = threadIdx.x & 31;
  const int piece_end = min(n, (i / kEmbSeg + 1) * kEmbSeg);
  const long long key = keys[i], k_before = keys[max(i - 1, 0)], k_next = keys[min(i + 1, n - 1)];
  int src = static_cast<int>(order[i]);
  int len = 1;
  const bool from_left = i > 0 && k_before == key;
  if (from_left && i % kEmbSeg != 0) return;
  if (i + 1 < piece_end && k_next == key) {  // most ids stand alone and need none of this
    const int at = min(i + lane, n - 1);
    const unsigned different = ~__ballot_sync(0xffffffffu, i + lane < piece_end && keys[at] == key);
    len = different == 0u ? 32 : __ffs(different) - 1;
    src = static_cast<int>(order[at]);
  }
  const bool goes_on = i + len == piece_end && piece_end < n && keys[piece_end] == key;
  const bool whole = !from_left && !goes_on;
  float* out = whole ? main + key * H : partial + (i / kEmbSeg * 2ll + (from_left ? 0 : 1)) * H;
  for (int c0 = (threadIdx.x & ~31) * 8; c0 < H; c0 += blockDim.x * 8) {  // whole warps, for the shuffles
    const int c = c0 + lane * 8;
    const bool on = c < H;
    float4* m = reinterpret_cast<float4*>(out + c);
    float4 m0 = make_float4(0.f, 0.f, 0.f, 0.f), m1 = m0;
    if (on && whole) {
      m0 = m[0];
      m1 = m[1];
    }
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < len; j += 2) {
      uint4 v[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const long long row = __shfl_sync(0xffffffffu, src, (j + q) & 31);
        if (on && j + q < len) v[q] = *reinterpret_cast<const uint4*>(dy + row * H + c);
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (on && j + q < len) {
          float f[8];
          unpack8(v[q], f);
#pragma unroll
          for (int x = 0; x < 8; ++x) acc[x] += f[x];
        }
      }
    }
    if (on) {
      m[0] = make_float4(m0.x + acc[0], m0.y + acc[1], m0.z + acc[2], m0.w + acc[3]);
      m[1] = make_float4(m1.x + acc[4], m1.y + acc[5], m1.z + acc[6], m1.w + acc[7]);
    }
  }
}

// The runs that cross a multiple of kEmbSeg: main[key] += the sums of their pieces, in order.  A CTA looks through eight
// pieces for runs that start there and go on and takes 128 columns of each; its eight warps add an eighth of a run's
// pieces each, so that a run of 16384 equal ids is 64 additions deep.
constexpr int kEmbJoin = 8;
__global__ void __launch_bounds__(256) embedding_grad_join_kernel(const long long* keys,
                                                                  const float* partial,
                                                                  float* main, long long n, int H) {
  chain_wait();
  chain_trigger();
  __shared__ float4 sums[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.y * 128 + lane * 4;
  const long long p0 = static_cast<long long>(blockIdx.x) * kEmbJoin;
  bool mine = false;
  if (lane < kEmbJoin && (p0 + lane + 1) * kEmbSeg < n) {
    const long long first = (p0 + lane) * kEmbSeg, next = first + kEmbSeg;
    const long long key = keys[next];
    mine = keys[next - 1] == key && !(first > 0 && keys[first - 1] == key);
  }
  for (unsigned todo = __ballot_sync(0xffffffffu, mine); todo != 0u; todo &= todo - 1u) {  // the same in every warp
    const long long p = p0 + __ffs(todo) - 1;
    const long long key = keys[(p + 1) * kEmbSeg];
    long long count = 1;  // pieces of the run: those behind p whose first position still belongs to it, 32 at a time
    for (unsigned on = ~0u; on == ~0u;) {
      const long long q = (p + count + lane) * kEmbSeg;
      on = __ballot_sync(0xffffffffu, q < n && keys[min(q, n - 1)] == key);
      count += on == ~0u ? 32 : __ffs(~on) - 1;
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < H) {
#pragma unroll 8
      for (long long s = count * warp / 8; s < count * (warp + 1) / 8; ++s) {
        const float4 v = *reinterpret_cast<const float4*>(partial + ((p + s) * 2 + (s == 0 ? 1 : 0)) * H + c);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
    }
    sums[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && c < H) {
      for (int w = 1; w < 8; ++w) {
        const float4 v = sums[w][lane];
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      float4* m = reinterpret_cast<float4*>(main + key * H + c);
      const float4 v = *m;
      *m = make_float4(v.x + acc.x, v.y + acc.y, v.z + acc.z, v.w + acc.w);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------ gather / combine
__global__ void gather_rows_kernel(const __nv_bfloat16* src, const int* row_slot,
                                   int slot_div, const float* slot_scale,
                                   __nv_bfloat16* out, long long cap_rows,
                                   const int* num_m_tiles, int H, long long ld_src, long long ld_out) {
  chain_wait();
  chain_trigger();
  const long long n_rows = num_m_tiles ? min(static_cast<long long>(*num_m_tiles) * 128, cap_rows) : cap_rows;
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long r = blockIdx.x * static_cast<long long>(warps_per_block) + (threadIdx.x >> 5); r < n_rows;
       r += static_cast<long long>(gridDim.x) * warps_per_block) {
    const int slot = row_slot[r];
    __nv_bfloat16* o = out + r * ld_out;
    if (slot < 0) {
      for (int c = lane * 8; c < H; c += 256) *reinterpret_cast<uint4*>(o + c) = make_uint4(0u, 0u, 0u, 0u);
    } else {
      const __nv_bfloat16* s = src + static_cast<long long>(slot / slot_div) * ld_src;
      const float sc = slot_scale != nullptr ? slot_scale[slot] : 1.f;
      for (int c = lane * 8; c < H; c += 1024) {  // four loads in flight, all ahead of the first store
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c + q * 256 < H) v[q] = *reinterpret_cast<const uint4*>(s + c + q * 256);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (c + q * 256 >= H) continue;
          if (slot_scale == nullptr) {
            *reinterpret_cast<uint4*>(o + c + q * 256) = v[q];
          } else {
            float f[8];
            unpack8(v[q], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] *= sc;
            store8(o + c + q * 256, f);
          }
        }
      }
    }
  }
}

// The same rows without a scale, token by token: a warp loads 1024 columns of a token's row once and stores them at all K
// places.  What bounds it: the stores (a plain zero fill writes at 5.8 TB/s here).  Row by row in expert order, a token is
// read K times, and between those reads the stream of stores has driven it out of L2.  Row by row / this, behind GEMMs:
// 16384 tokens x 2048 columns, top-8 of 64: 174 / 122 us; 3333 x 4096, top-8 of 32: 68 / 56; 8192 x 4096, top-2 of 8:
// 48 / 40; 16384 x 512, top-1 of 16: 15.3 / 13.2; 16384 x 4096, top-1 of 8: 52 / 52.  (Bulk copies through shared memory
// instead of registers: 130, 67, 57, 22, 67.)
// Few tokens leave mostly padding to write, up to 127 rows per expert, so it has warps of its own, kPadRows rows each, that
// run beside the tokens'.  By the tokens' warps behind their rows it took longer than row by row: 64 x 2048, top-8 of 64
// 11.8 us in a loop against 6.4, 1000 tokens 18.5 / 9.3; this way 9.8 and 13.3 there, and with a buffer that is not in L2,
// as a new one, as long as row by row (12 and 15 us).  In a layer's forward and backward, whose first GEMM loads weights
// meanwhile, 0.4 to 1 us less than behind the rows; 1, 4 and 16 rows per warp 700, 699 and 698 us for 64 tokens of E 64 H
// 2048 F 1024, 805, 804 and 806 for 1000.
constexpr int kPadRows = 4;
__global__ void place_rows_kernel(const PlaceRowsArgs a, int pieces) {
  chain_wait();
  chain_trigger();
  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.src);
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out);
  const int lane = threadIdx.x & 31;
  const long long first = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const long long step = (gridDim.x * static_cast<long long>(blockDim.x)) >> 5;
  const long long items = (a.n_tokens + (a.zero_padding ? a.n_local * (128LL / kPadRows) : 0)) * pieces;
  for (long long it = first; it < items; it += step) {
    const long long t = it / pieces;
    const int c0 = static_cast<int>(it - t * pieces) * 1024 + lane * 8;
    if (t >= a.n_tokens) {  // rows of padding behind an expert's rows
      const int i = static_cast<int>(t - a.n_tokens), e = i / (128 / kPadRows);
      const long long row = static_cast<long long>(a.group_offsets[e]) + a.counts_kept[e] + i % (128 / kPadRows) * kPadRows;
      const int end = a.group_offsets[e + 1];
#pragma unroll
      for (int r = 0; r < kPadRows; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (row + r < end && c0 + q * 256 < a.H)
            *reinterpret_cast<uint4*>(out + (row + r) * a.ld_out + c0 + q * 256) = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const __nv_bfloat16* s = src + t * a.ld_src + c0;
    uint4 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c0 + q * 256 < a.H) v[q] = *reinterpret_cast<const uint4*>(s + q * 256);
    for (int k0 = 0; k0 < a.K; k0 += 32) {
      const int mine = k0 + lane < a.K ? a.slot_row[t * a.K + k0 + lane] : -1;
      const int n = min(32, a.K - k0);
      for (int k = 0; k < n; ++k) {
        const int row = __shfl_sync(0xffffffffu, mine, k);
        if (row < 0) continue;  // dropped
        __nv_bfloat16* o = out + row * a.ld_out + c0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c0 + q * 256 < a.H) *reinterpret_cast<uint4*>(o + q * 256) = v[q];
      }
    }
  }
}

__global__ void combine_rows_kernel(const __nv_bfloat16* rows, const int* slot_row,
                                    const float* w, __nv_bfloat16* y, long long n_tokens,
                                    int K, int H, long long ld_rows, long long ld_y) {
  chain_wait();
  chain_trigger();
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long t = blockIdx.x * static_cast<long long>(warps_per_block) + (threadIdx.x >> 5); t < n_tokens;
       t += static_cast<long long>(gridDim.x) * warps_per_block) {
    for (int c = lane * 8; c < H; c += 256) {
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
      for (int k = 0; k < K; ++k) {
        const int r = slot_row[t * K + k];
        if (r < 0) continue;
        const float wk = w ? w[t * K + k] : 1.f;
        float f[8];
        load8(rows + static_cast<long long>(r) * ld_rows + c, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += wk * f[j];
      }
      store8(y + t * ld_y + c, acc);
    }
  }
}

// Same sum for a compile-time K: the K (row, weight) pairs of a token are looked up once (lane k loads pair k, the
// warp shares them by shuffle) and the loads of all K rows of a column block are issued before the first use, so a
// lane keeps K x 16 bytes in flight instead of 16.  The order of the additions is that of the kernel above.  Few
// tokens are cut into pieces of columns (multiples of 256), one per warp, until the warps fill the GPU: a warp that
// walks a row of 2048 columns alone waits eight times for memory (64 tokens, top-8: 10.4 us).
template <int KK>
__global__ void combine_rows_k_kernel(const __nv_bfloat16* rows, const int* slot_row,
                                      const float* w, __nv_bfloat16* y, long long n_tokens,
                                      int H, long long ld_rows, long long ld_y, int pieces, int piece_cols) {
  chain_wait();
  chain_trigger();
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long i = blockIdx.x * static_cast<long long>(warps_per_block) + (threadIdx.x >> 5); i < n_tokens * pieces;
       i += static_cast<long long>(gridDim.x) * warps_per_block) {
    const long long t = pieces == 1 ? i : i / pieces;
    const int c0 = pieces == 1 ? 0 : static_cast<int>(i - t * pieces) * piece_cols;
    const int c1 = min(H, c0 + piece_cols);
    int my_r = -1;
    float my_w = 0.f;
    if (lane < KK) {
      my_r = slot_row[t * KK + lane];
      my_w = w ? w[t * KK + lane] : 1.f;
    }
    const __nv_bfloat16* src[KK];
    float wk[KK];
#pragma unroll
    for (int k = 0; k < KK; ++k) {
      const int r = __shfl_sync(0xffffffffu, my_r, k);
      wk[k] = __shfl_sync(0xffffffffu, my_w, k);
      src[k] = r >= 0 ? rows + static_cast<long long>(r) * ld_rows : nullptr;
    }
    for (int c = c0 + lane * 8; c < c1; c += 256) {
      uint4 v[KK];
#pragma unroll
      for (int k = 0; k < KK; ++k)
        v[k] = src[k] != nullptr ? *reinterpret_cast<const uint4*>(src[k] + c) : make_uint4(0u, 0u, 0u, 0u);
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
      for (int k = 0; k < KK; ++k) {
        if (src[k] == nullptr) continue;  // a dropped slot adds nothing (and no signed zero)
        const float2 a = unpack_bf16x2(v[k].x), b = unpack_bf16x2(v[k].y), cc = unpack_bf16x2(v[k].z),
                     d = unpack_bf16x2(v[k].w);
        acc[0] += wk[k] * a.x; acc[1] += wk[k] * a.y; acc[2] += wk[k] * b.x; acc[3] += wk[k] * b.y;
        acc[4] += wk[k] * cc.x; acc[5] += wk[k] * cc.y; acc[6] += wk[k] * d.x; acc[7] += wk[k] * d.y;
      }
      store8(y + t * ld_y + c, acc);
    }
  }
}

__global__ void combine_bwd_w_kernel(const __nv_bfloat16* rows, const int* slot_row,
                                     const __nv_bfloat16* dy, float* dw, long long n_tokens,
                                     int K, int H, long long ld_rows, long long ld_dy) {
  chain_wait();
  chain_trigger();
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long n_slots = n_tokens * K;
  for (long long s = blockIdx.x * static_cast<long long>(warps_per_block) + (threadIdx.x >> 5); s < n_slots;
       s += static_cast<long long>(gridDim.x) * warps_per_block) {
    const int r = slot_row[s];
    float acc = 0.f;
    if (r >= 0) {
      const __nv_bfloat16* a = rows + static_cast<long long>(r) * ld_rows;
      const __nv_bfloat16* b = dy + (s / K) * ld_dy;
      for (int c = lane * 8; c < H; c += 256) {
        float fa[8], fb[8];
        load8(a + c, fa);
        load8(b + c, fb);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc += fa[j] * fb[j];
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) dw[s] = acc;
  }
}

// Backward of the weighted combine, token by token: a warp holds the token's row of dy, multiplies it by each pick's weight
// into the expert's row, and takes its product with that pick's result row, which is the gradient of the weight.  What
// bounds it: reading the result rows and writing as many.  In two launches (combine_bwd_w, then gather_rows with a scale) dy
// was read K times for each, in between the stores that drive it out of L2.  The values and the order of every sum are
// theirs.  Both / this, behind GEMMs: 16384 tokens x 2048, top-8 of 64 286 / 192 us (1.2 GB: 175 at the copy rate);
// 3333 x 4096, top-8 of 32 120 / 93; 8192 x 4096, top-2 of 8 85 / 75; 4096 x 1024, top-2 of 16 21.5 / 17.4; 16384 x 512,
// top-1 of 16 23.6 / 17.4.  Q: 16-byte pieces of dy per lane, H <= 256 Q; wider rows keep the two launches.
// Few tokens are 2^split_log2 warps each, which share the token's picks: one warp's picks follow one another, each behind
// its reads.  Rows in L2, two launches / one warp per token / this: 64 x 2048, top-8 of 64 9.4 / 11.6 / 6.7 us, 500 tokens
// 11.6 / 13.4 / 8.3, 1000 18.3 / 15.2 / 11.1; 64 x 4096, top-8 of 32 11.4 / 14.6 / 7.6; 1000 x 1024, top-2 of 16 5.2 / 4.0
// / 3.0.
template <int Q>
__global__ void __launch_bounds__(256) combine_grad_kernel(const PlaceRowsArgs a, const float* weight,
                                                           const __nv_bfloat16* rows, long long ld_rows, float* dw,
                                                           int split_log2) {
  chain_wait();
  chain_trigger();
  const __nv_bfloat16* dy = static_cast<const __nv_bfloat16*>(a.src);
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out);
  const int lane = threadIdx.x & 31;
  const long long warp = (blockIdx.x * 256LL + threadIdx.x) >> 5;
  const long long workers = a.n_tokens << split_log2;
  if (warp < workers) {
    const long long t = warp >> split_log2;
    uint4 d[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (lane * 8 + q * 256 < a.H) d[q] = *reinterpret_cast<const uint4*>(dy + t * a.ld_src + lane * 8 + q * 256);
    for (int k = static_cast<int>(warp - (t << split_log2)); k < a.K; k += 1 << split_log2) {
      const long long slot = t * a.K + k;
      const int row = a.slot_row[slot];
      float acc = 0.f;
      if (row >= 0) {
        uint4 y[Q];
        if (dw != nullptr) {
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if (lane * 8 + q * 256 < a.H)
              y[q] = *reinterpret_cast<const uint4*>(rows + row * ld_rows + lane * 8 + q * 256);
        }
        const float w = weight[slot];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          if (lane * 8 + q * 256 >= a.H) continue;
          float f[8], s[8];
          unpack8(d[q], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] = f[j] * w;
          store8(out + row * a.ld_out + lane * 8 + q * 256, s);
          if (dw != nullptr) {
            float g[8];
            unpack8(y[q], g);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc += g[j] * f[j];
          }
        }
      }
      if (dw != nullptr) {
        acc = warp_sum(acc);
        if (lane == 0) dw[slot] = acc;  // 0 for a dropped slot
      }
    }
    return;
  }
  // the warps behind the tokens': an expert's rows are followed by up to 127 rows of padding
  const long long i = warp - workers;
  if (i >= a.n_local * 128LL) return;
  const int e = static_cast<int>(i >> 7);
  const long long row = static_cast<long long>(a.group_offsets[e]) + a.counts_kept[e] + (i & 127);
  if (row < a.group_offsets[e + 1])
    for (int c = lane * 8; c < a.H; c += 256) *reinterpret_cast<uint4*>(out + row * a.ld_out + c) = make_uint4(0u, 0u, 0u, 0u);
}

inline unsigned grid_for(long long work_items, int per_block, int max_blocks) {
  long long b = (work_items + per_block - 1) / per_block;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return static_cast<unsigned>(b);
}

}  // namespace

inline int rn_vec_for(int H) {
  const int per = RN_THREADS * 8;
  const int need = (H + per - 1) / per;
  return need <= 1 ? 1 : need <= 2 ? 2 : need <= 4 ? 4 : 8;
}

cudaError_t launch_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, long long rows, int H, float eps,
                               cudaStream_t stream, const void* delta, void* sum) {
  if (H % 8 != 0 || H > RN_THREADS * 8 * 8 || rows <= 0) return cudaErrorInvalidValue;
  const unsigned grid = grid_for(rows, 1, 148 * 32);
  auto go = [&](auto add, auto plain) {
    launch_chained(delta != nullptr ? add : plain, grid, RN_THREADS, 0, stream, reinterpret_cast<const __nv_bfloat16*>(x),
                   reinterpret_cast<const __nv_bfloat16*>(delta), reinterpret_cast<__nv_bfloat16*>(sum),
                   reinterpret_cast<const __nv_bfloat16*>(w), reinterpret_cast<__nv_bfloat16*>(y), rstd, rows, H, eps);
  };
  switch (rn_vec_for(H)) {
    case 1: go(rmsnorm_fwd_kernel<1, true>, rmsnorm_fwd_kernel<1, false>); break;
    case 2: go(rmsnorm_fwd_kernel<2, true>, rmsnorm_fwd_kernel<2, false>); break;
    case 4: go(rmsnorm_fwd_kernel<4, true>, rmsnorm_fwd_kernel<4, false>); break;
    default: go(rmsnorm_fwd_kernel<8, true>, rmsnorm_fwd_kernel<8, false>); break;
  }
  return cudaGetLastError();
}

long long rmsnorm_bwd_partial_rows(long long rows, int num_sms) {
  return grid_for(rows, 1, (num_sms > 0 ? num_sms : 148) * 4);  // one wave of persistent CTAs
}

template <int VEC, bool RES>
static cudaError_t launch_rmsnorm_bwd_variant(const void* dy, const void* dres, const void* x, const void* w,
                                              const float* rstd, void* dx, float* dw, float* dw_partial, long long rows,
                                              int H, unsigned grid, cudaStream_t stream) {
  constexpr int smem = rn_bwd_smem(VEC, RES ? 3 : 2);
  if (smem + 1024 > 48 * 1024) {  // static shared memory counts too; asked for on the device that launches
    const cudaError_t e =
        cudaFuncSetAttribute(rmsnorm_bwd_kernel<VEC, RES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(rmsnorm_bwd_kernel<VEC, RES>, grid, RN_THREADS, smem, stream,
                        reinterpret_cast<const __nv_bfloat16*>(dy), reinterpret_cast<const __nv_bfloat16*>(dres),
                        reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(w), rstd,
                        reinterpret_cast<__nv_bfloat16*>(dx), dw, dw_partial, rows, H);
}

cudaError_t launch_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx, float* dw,
                               float* dw_partial, long long rows, int H, int num_sms, cudaStream_t stream,
                               const void* dres) {
  if (H % 8 != 0 || H > RN_THREADS * 8 * 8 || rows <= 0) return cudaErrorInvalidValue;
  const unsigned grid = static_cast<unsigned>(rmsnorm_bwd_partial_rows(rows, num_sms));
  if (dw == nullptr) dw_partial = nullptr;
  auto go = [&](auto res, auto plain) {
    return (dres != nullptr ? res : plain)(dy, dres, x, w, rstd, dx, dw, dw_partial, rows, H, grid, stream);
  };
  cudaError_t e;
  switch (rn_vec_for(H)) {
    case 1: e = go(launch_rmsnorm_bwd_variant<1, true>, launch_rmsnorm_bwd_variant<1, false>); break;
    case 2: e = go(launch_rmsnorm_bwd_variant<2, true>, launch_rmsnorm_bwd_variant<2, false>); break;
    case 4: e = go(launch_rmsnorm_bwd_variant<4, true>, launch_rmsnorm_bwd_variant<4, false>); break;
    default: e = go(launch_rmsnorm_bwd_variant<8, true>, launch_rmsnorm_bwd_variant<8, false>); break;
  }
  if (e == cudaSuccess && dw_partial != nullptr)
    e = launch_chained(colsum_kernel, (H + 31) / 32, CSUM_WARPS * 32, 0, stream, dw_partial, dw, static_cast<int>(grid), H);
  return e;
}

cudaError_t launch_rope(void* t, const float* cos_tab, const float* sin_tab, long long rows, int seq, int heads,
                        int head_dim, long long row_stride, int inverse, cudaStream_t stream) {
  if (head_dim % 16 != 0 || rows <= 0) return cudaErrorInvalidValue;
  const long long total = rows * heads * (head_dim / 16);
  launch_chained(rope_kernel, grid_for(total, 256, 148 * 16), 256, 0, stream, reinterpret_cast<__nv_bfloat16*>(t),
                 cos_tab, sin_tab, rows, seq, heads, head_dim, row_stride, inverse);
  return cudaGetLastError();
}

cudaError_t launch_qkv_grad_pack(const void* dq, const long long* dq_strides, const void* dk, const long long* dk_strides,
                                 const void* dv, const long long* dv_strides, void* out, const float* cos_tab,
                                 const float* sin_tab, long long batch, int seq, int nh, int nkv, int head_dim,
                                 cudaStream_t stream) {
  if (head_dim % 16 != 0 || batch <= 0 || seq <= 0 || nh <= 0 || nkv <= 0) return cudaErrorInvalidValue;
  auto mk = [](const void* p, const long long* st) {
    return QkvGradSrc{reinterpret_cast<const __nv_bfloat16*>(p), st[0], st[1], st[2]};
  };
  for (const long long* st : {dq_strides, dk_strides, dv_strides})
    if (st[0] % 8 != 0 || st[1] % 8 != 0 || st[2] % 8 != 0) return cudaErrorInvalidValue;  // 16-byte vector loads
  const long long rows = batch * seq;
  const long long total = rows * (nh + 2 * nkv) * (head_dim / 16);
  launch_chained(qkv_grad_pack_kernel, grid_for(total, 256, 148 * 16), 256, 0, stream, mk(dq, dq_strides), mk(dk,
                 dk_strides), mk(dv, dv_strides), reinterpret_cast<__nv_bfloat16*>(out), cos_tab, sin_tab, rows, seq,
                 nh, nkv, head_dim);
  return cudaGetLastError();
}

cudaError_t launch_adamw(const AdamWArgs& a, cudaStream_t stream) {
  if (a.n <= 0) return cudaSuccess;
  const auto on32 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 32 == 0; };
  const long long blocks = (a.n / 8 + 255) / 256;
  if (!a.grad_is_bf16 && a.n % 8 == 0 && on32(a.p32) && on32(a.m) && on32(a.v) && on32(a.grad) &&
      reinterpret_cast<uintptr_t>(a.p16) % 16 == 0 && blocks <= INT_MAX)
    launch_chained(adamw_wide_kernel, static_cast<unsigned>(blocks), 256, 0, stream, a);
  else
    launch_chained(adamw_kernel, grid_for(a.n / 4 + 1, 256, 148 * 16), 256, 0, stream, a);
  return cudaGetLastError();
}

int sumsq_partial_count(long long n) { return n <= 0 ? 0 : static_cast<int>(grid_for(n / 8 + 1, 256, 148 * 8)); }

cudaError_t launch_sumsq(const void* x, int is_bf16, long long n, float* out, float* partials, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const unsigned grid = static_cast<unsigned>(sumsq_partial_count(n));
  launch_chained(sumsq_kernel, grid, 256, 0, stream, x, is_bf16, n, out, partials);
  if (partials != nullptr) launch_chained(sumsq_final_kernel, 1, 256, 0, stream, partials, static_cast<int>(grid), out);
  return cudaGetLastError();
}

cudaError_t launch_splitk_reduce(const float* part, int parts, long long n, void* out, int out_bf16, int accumulate,
                                 cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (n % 4 != 0 || parts < 1 || (out_bf16 && accumulate)) return cudaErrorInvalidValue;
  const long long n4 = n / 4;
  const unsigned grid = static_cast<unsigned>((n4 + 255) / 256);
  const float4* p = reinterpret_cast<const float4*>(part);
  if (out_bf16) launch_chained(splitk_reduce_kernel<2>, grid, 256, 0, stream, p, parts, n4, out);
  else if (accumulate) launch_chained(splitk_reduce_kernel<1>, grid, 256, 0, stream, p, parts, n4, out);
  else launch_chained(splitk_reduce_kernel<0>, grid, 256, 0, stream, p, parts, n4, out);
  return cudaGetLastError();
}

cudaError_t launch_scaled_out(const float* x, const float* scale, long long n, void* out, int out_bf16, int accumulate,
                              cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (n % 4 != 0 || (out_bf16 && accumulate)) return cudaErrorInvalidValue;
  const long long n4 = n / 4;
  const unsigned grid = static_cast<unsigned>((n4 + 1023) / 1024);
  const float4* x4 = reinterpret_cast<const float4*>(x);
  if (out_bf16) return launch_chained(scaled_out_kernel<2>, grid, 256, 0, stream, x4, scale, n4, out);
  if (accumulate) return launch_chained(scaled_out_kernel<1>, grid, 256, 0, stream, x4, scale, n4, out);
  return launch_chained(scaled_out_kernel<0>, grid, 256, 0, stream, x4, scale, n4, out);
}

cudaError_t launch_scaled_bf16(const void* x, const float* scale, long long n, void* out, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (n % 8 != 0) return cudaErrorInvalidValue;
  return launch_chained(scaled_bf16_kernel, static_cast<unsigned>((n / 8 + 1023) / 1024), 256, 0, stream,
                        reinterpret_cast<const uint4*>(x), scale, n / 8, reinterpret_cast<uint4*>(out));
}

long long embedding_grad_partial_floats(long long n, int H) {
  return n <= kEmbSeg ? 0 : (n + kEmbSeg - 1) / kEmbSeg * 2 * H;
}

cudaError_t launch_embedding_grad(const void* dy, const long long* keys, const long long* order, float* main,
                                  float* partial, long long n, int H, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (H % 8 != 0 || n > INT_MAX - kEmbSeg || (n > kEmbSeg && partial == nullptr)) return cudaErrorInvalidValue;
  const int threads = H / 8 >= 256 ? 256 : (H / 8 + 31) / 32 * 32;
  const cudaError_t e = launch_chained(embedding_grad_kernel, static_cast<unsigned>(n), threads, 0, stream,
                                       reinterpret_cast<const __nv_bfloat16*>(dy), keys, order, main, partial,
                                       static_cast<int>(n), H);
  if (e != cudaSuccess || n <= kEmbSeg) return e;
  const long long pieces = (n + kEmbSeg - 1) / kEmbSeg;
  return launch_chained(embedding_grad_join_kernel, dim3(static_cast<unsigned>((pieces + kEmbJoin - 1) / kEmbJoin), (H + 127) / 128), 256,
                        0, stream, keys, partial, main, n, H);
}

cudaError_t launch_cross_entropy(void* logits, const float2* stats, const long long* targets, float* loss_sum,
                                 float* row_loss, long long rows, int V, long long ld, float grad_scale,
                                 cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  if (ld % 8 != 0) return cudaErrorInvalidValue;
  auto lb = reinterpret_cast<__nv_bfloat16*>(logits);
  if (stats != nullptr && V % 8 == 0)
    launch_chained(cross_entropy_stats_kernel, static_cast<unsigned>(rows), CS_THREADS, 0, stream, lb, stats, targets,
                   loss_sum, row_loss, V, ld, grad_scale);
  else
    launch_chained(cross_entropy_kernel, static_cast<unsigned>(rows), CE_THREADS, 0, stream, lb, targets, loss_sum, row_loss,
                   rows, V, ld, grad_scale);
  return cudaGetLastError();
}

cudaError_t launch_gather_rows(const void* src, const int* row_slot, int slot_div, const float* slot_scale, void* out,
                               long long cap_rows, const int* num_m_tiles, int H, long long ld_src, long long ld_out,
                               cudaStream_t stream) {
  if (H % 8 != 0 || cap_rows <= 0 || slot_div <= 0) return cudaErrorInvalidValue;
  launch_chained(gather_rows_kernel, grid_for(cap_rows, 8, 148 * 8), 256, 0, stream,
                 reinterpret_cast<const __nv_bfloat16*>(src), row_slot, slot_div, slot_scale,
                 reinterpret_cast<__nv_bfloat16*>(out), cap_rows, num_m_tiles, H, ld_src, ld_out);
  return cudaGetLastError();
}

cudaError_t launch_place_rows(const PlaceRowsArgs& a, cudaStream_t stream) {
  if (a.H % 8 != 0 || a.H <= 0 || a.K <= 0) return cudaErrorInvalidValue;
  if (a.n_tokens <= 0) return cudaSuccess;
  const int pieces = (a.H + 1023) / 1024;
  const long long warps = (a.n_tokens + (a.zero_padding ? a.n_local * (128LL / kPadRows) : 0)) * pieces;
  // a warp per piece: CTAs that stride over the tokens drift apart (16384 x 2048, top-8: 130 / 120 us)
  launch_chained(place_rows_kernel, grid_for(warps, 8, 1 << 24), 256, 0, stream, a, pieces);
  return cudaGetLastError();
}

bool combine_grad_supported(int H) { return H <= 4096; }
cudaError_t launch_combine_grad(const PlaceRowsArgs& a, const float* weight, const void* rows, long long ld_rows, float* dw,
                                cudaStream_t stream) {
  if (a.H % 8 != 0 || a.H <= 0 || !combine_grad_supported(a.H) || a.K <= 0 || a.n_tokens <= 0) return cudaErrorInvalidValue;
  // Shared as long as the chip is not full of warps with a row of dy each, which several would read for nothing: 6 MB of
  // them, 40 KB per SM.  2000 x 2048, top-8 of 64: 25.6 us with one warp per token, 26.8 with two, 28.1 with four; 800 x
  // 4096, top-8 of 32: 24.6, 25.7, 26.4; 2000 x 512, top-4 of 16: 5.4, 4.2, 4.1.
  int split_log2 = 0;
  while ((2 << split_log2) <= a.K && (a.n_tokens << split_log2) * a.H < (3LL << 20)) ++split_log2;
  const unsigned grid = grid_for((a.n_tokens << split_log2) + a.n_local * 128LL, 8, INT_MAX);
  const int q = (a.H + 255) / 256;
  auto go = [&](auto kernel) {
    return launch_chained(kernel, grid, 256, 0, stream, a, weight, reinterpret_cast<const __nv_bfloat16*>(rows), ld_rows, dw,
                          split_log2);
  };
  return q <= 2 ? go(combine_grad_kernel<2>) : q <= 4 ? go(combine_grad_kernel<4>)
       : q <= 8 ? go(combine_grad_kernel<8>) : go(combine_grad_kernel<16>);
}

cudaError_t launch_combine_rows(const void* rows, const int* slot_row, const float* w, void* y, long long n_tokens,
                                int K, int H, long long ld_rows, long long ld_y, cudaStream_t stream) {
  if (H % 8 != 0 || n_tokens <= 0) return cudaErrorInvalidValue;
  static const bool generic_only = [] {
    const char* v = std::getenv("CMOE_COMBINE_GENERIC");  // A/B switch: the kernel with a run-time K for every K
    return v != nullptr && v[0] != '\0' && v[0] != '0';
  }();
  if (!generic_only && (K == 8 || K == 6 || K == 4 || K == 2)) {
    const long long want = 148 * 32 / n_tokens, blocks256 = (H + 255) / 256;
    const int piece_cols = static_cast<int>(want <= 1 ? blocks256 : (blocks256 + want - 1) / want) * 256;
    const int pieces = (H + piece_cols - 1) / piece_cols;
    const unsigned grid = grid_for(n_tokens * pieces, 8, 148 * 8);
    auto rb = reinterpret_cast<const __nv_bfloat16*>(rows);
    auto yb = reinterpret_cast<__nv_bfloat16*>(y);
    switch (K) {
      case 8: launch_chained(combine_rows_k_kernel<8>, grid, 256, 0, stream, rb, slot_row, w, yb, n_tokens, H,
                             ld_rows, ld_y, pieces, piece_cols); break;
      case 6: launch_chained(combine_rows_k_kernel<6>, grid, 256, 0, stream, rb, slot_row, w, yb, n_tokens, H,
                             ld_rows, ld_y, pieces, piece_cols); break;
      case 4: launch_chained(combine_rows_k_kernel<4>, grid, 256, 0, stream, rb, slot_row, w, yb, n_tokens, H,
                             ld_rows, ld_y, pieces, piece_cols); break;
      default: launch_chained(combine_rows_k_kernel<2>, grid, 256, 0, stream, rb, slot_row, w, yb, n_tokens, H,
                              ld_rows, ld_y, pieces, piece_cols); break;
    }
    return cudaGetLastError();
  }
  launch_chained(combine_rows_kernel, grid_for(n_tokens, 8, 148 * 8), 256, 0, stream,
                 reinterpret_cast<const __nv_bfloat16*>(rows), slot_row, w, reinterpret_cast<__nv_bfloat16*>(y),
                 n_tokens, K, H, ld_rows, ld_y);
  return cudaGetLastError();
}

cudaError_t launch_combine_bwd_w(const void* rows, const int* slot_row, const void* dy, float* dw, long long n_tokens,
                                 int K, int H, long long ld_rows, long long ld_dy, cudaStream_t stream) {
  if (H % 8 != 0 || n_tokens <= 0) return cudaErrorInvalidValue;
  launch_chained(combine_bwd_w_kernel, grid_for(n_tokens * K, 8, 148 * 8), 256, 0, stream,
                 reinterpret_cast<const __nv_bfloat16*>(rows), slot_row, reinterpret_cast<const __nv_bfloat16*>(dy),
                 dw, n_tokens, K, H, ld_rows, ld_dy);
  return cudaGetLastError();
}

}  // namespace cmoe
