// Element math of the SwiGLU epilogues, shared by the one-SM and the two-SM GEMM.
#pragma once
#include "common.cuh"

namespace cmoe {

// ex2.approx + rcp.approx: two special-function instructions instead of an IEEE division (the epilogue warps are
// issue-bound: one warp per scheduler, so every instruction saved per element shortens the tile)
__device__ __forceinline__ float sigmoidf_fast(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }

// SwiGLU backward for 32 columns of one row: dH (fp32 bits in r) with the saved gate / up values (bf16, packed in
// cg / cu) -> dGate / dUp (bf16, packed) written over cg / cu.  Eight columns at a time, straight from the packed
// inputs to the packed outputs.
// WEIGHTED: the forward multiplied h by the row's weight w, and r holds the gradient of that product.  The gradients of
// gate and up take the factor w, and `dot` the row's share of the weight's own gradient, sum of r * silu(gate) * up over
// the first `live` groups of eight columns.  What it costs: 3 of some 25 instructions per element.
template <bool WEIGHTED>
__device__ __forceinline__ void swiglu_bwd_math(const uint32_t (&r)[32], uint4 (&cg)[4], uint4 (&cu)[4], float w, int live,
                                                float& dot) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t gw[4] = {cg[j].x, cg[j].y, cg[j].z, cg[j].w};
    const uint32_t uw[4] = {cu[j].x, cu[j].y, cu[j].z, cu[j].w};
    uint32_t og[4], ou[4];
    float part = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 g = unpack_bf16x2(gw[q]);
      const float2 u = unpack_bf16x2(uw[q]);
      const float dh0 = __uint_as_float(r[8 * j + 2 * q]), dh1 = __uint_as_float(r[8 * j + 2 * q + 1]);
      const float s0 = sigmoidf_fast(g.x), s1 = sigmoidf_fast(g.y);
      // d silu(g)/dg = s (1 + g (1 - s))
      const float ds0 = s0 * fmaf(g.x, 1.f - s0, 1.f), ds1 = s1 * fmaf(g.y, 1.f - s1, 1.f);
      const float du0 = dh0 * (g.x * s0), du1 = dh1 * (g.y * s1);
      if (WEIGHTED) {
        part = fmaf(du0, u.x, part);
        part = fmaf(du1, u.y, part);
        og[q] = pack_bf16x2(w * dh0 * u.x * ds0, w * dh1 * u.y * ds1);
        ou[q] = pack_bf16x2(w * du0, w * du1);
      } else {
        og[q] = pack_bf16x2(dh0 * u.x * ds0, dh1 * u.y * ds1);
        ou[q] = pack_bf16x2(du0, du1);
      }
    }
    if (WEIGHTED && j < live) dot += part;
    cg[j] = make_uint4(og[0], og[1], og[2], og[3]);
    cu[j] = make_uint4(ou[0], ou[1], ou[2], ou[3]);
  }
}

// The weight of a row: of the slot that it came from, 0 for padding, 1 where rows have none.
__device__ __forceinline__ float row_weight(const int* row_slot, const float* slot_weight, long long row) {
  if (slot_weight == nullptr) return 1.f;
  const int slot = row_slot[row];
  return slot >= 0 ? slot_weight[slot] : 0.f;
}

}  // namespace cmoe
