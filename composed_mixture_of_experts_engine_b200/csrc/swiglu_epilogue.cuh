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
__device__ __forceinline__ void swiglu_bwd_math(const uint32_t (&r)[32], uint4 (&cg)[4], uint4 (&cu)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t gw[4] = {cg[j].x, cg[j].y, cg[j].z, cg[j].w};
    const uint32_t uw[4] = {cu[j].x, cu[j].y, cu[j].z, cu[j].w};
    uint32_t og[4], ou[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 g = unpack_bf16x2(gw[q]);
      const float2 u = unpack_bf16x2(uw[q]);
      const float dh0 = __uint_as_float(r[8 * j + 2 * q]), dh1 = __uint_as_float(r[8 * j + 2 * q + 1]);
      const float s0 = sigmoidf_fast(g.x), s1 = sigmoidf_fast(g.y);
      // d silu(g)/dg = s (1 + g (1 - s))
      const float dg0 = dh0 * u.x * (s0 * fmaf(g.x, 1.f - s0, 1.f));
      const float dg1 = dh1 * u.y * (s1 * fmaf(g.y, 1.f - s1, 1.f));
      og[q] = pack_bf16x2(dg0, dg1);
      ou[q] = pack_bf16x2(dh0 * (g.x * s0), dh1 * (g.y * s1));
    }
    cg[j] = make_uint4(og[0], og[1], og[2], og[3]);
    cu[j] = make_uint4(ou[0], ou[1], ou[2], ou[3]);
  }
}

}  // namespace cmoe
