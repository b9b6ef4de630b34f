// See tensor_maps.h.  A map is encoded on every call: the encoding is a host-side packing of its arguments and takes
// less time than a locked look-up by address and sizes did.
#include "tensor_maps.h"

#include <cstdint>
#include <mutex>

namespace cmoe {

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

cudaError_t encode(CUtensorMap* out, CUtensorMapDataType type, int rank, const void* ptr, const cuuint64_t* dims,
                   const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle,
                   CUtensorMapL2promotion promotion) {
  const EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return cudaErrorNotSupported;
  const cuuint32_t estride[3] = {1u, 1u, 1u};
  const auto pack = [&] {
    return enc(out, type, static_cast<cuuint32_t>(rank), const_cast<void*>(ptr), dims, strides, box, estride,
               CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (pack()) return cudaSuccess;
  // A thread that has made no runtime call yet (a backward thread whose first node this is) has no current context, which
  // the driver's encoder needs and cudaSetDevice brings.
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess && pack()) return cudaSuccess;
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t make_tmap(CUtensorMap* out, const void* ptr, long long rows, long long cols, long long ld, int box_rows,
                      int box_cols) {
  if ((box_cols != 64 && box_cols != 32) || (reinterpret_cast<uintptr_t>(ptr) & 15u) != 0 || (ld * 2) % 16 != 0 ||
      cols <= 0 || rows <= 0)
    return cudaErrorInvalidValue;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
  return encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, dims, strides, box,
                box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

cudaError_t make_tmap_out(CUtensorMap* out, const void* ptr, int fp32, long long groups, long long rows,
                          long long cols, long long ld, long long gstride, int box_bytes, int box_rows) {
  if (box_bytes != 128 && box_bytes != 64) return cudaErrorInvalidValue;
  const long long es = fp32 ? 4 : 2;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows),
                              static_cast<cuuint64_t>(groups)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld * es), static_cast<cuuint64_t>(gstride * es)};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(box_bytes / es), static_cast<cuuint32_t>(box_rows), 1u};
  return encode(out, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides,
                box, box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                CU_TENSOR_MAP_L2_PROMOTION_NONE);
}

cudaError_t make_tmap_halves(CUtensorMap* out, const void* ptr, long long rows, long long n, long long ld,
                             int box_rows) {
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(n), 2u, static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(n * 2), static_cast<cuuint64_t>(ld * 2)};
  const cuuint32_t box[3] = {32u, 1u, static_cast<cuuint32_t>(box_rows)};
  return encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B,
                CU_TENSOR_MAP_L2_PROMOTION_NONE);
}

}  // namespace cmoe
