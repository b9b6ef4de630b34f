// TMA descriptors of the GEMM and router kernels' operands and results.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace cmoe {

constexpr int kMapTileRows = 128;  // rows of one result piece

// bf16 row-major [rows, cols] (leading dimension ld), box = box_cols columns x box_rows rows; 64 columns use the
// 128-byte swizzle (operands), 32 columns the 64-byte swizzle (epilogue pieces)
cudaError_t make_tmap(CUtensorMap* out, const void* ptr, long long rows, long long cols, long long ld, int box_rows,
                      int box_cols = 64);
// Output map: [groups, rows, cols] of fp32 or bf16 with row stride ld and group stride gstride (elements); the box is
// one staging buffer, box_rows rows x box_bytes (128 or 64) bytes, in the swizzle of that width.
cudaError_t make_tmap_out(CUtensorMap* out, const void* ptr, int fp32, long long groups, long long rows,
                          long long cols, long long ld, long long gstride, int box_bytes = 128,
                          int box_rows = kMapTileRows);
// bf16 [rows, 2N] viewed as [rows, 2 halves, N] (gate | up): dims (N, 2, rows), box 32 columns x 1 half x box_rows rows,
// 64-byte swizzle; a store of columns [c, c+32) of one half is clipped at N and never reaches into the other half
cudaError_t make_tmap_halves(CUtensorMap* out, const void* ptr, long long rows, long long n, long long ld,
                             int box_rows = kMapTileRows);

}  // namespace cmoe
