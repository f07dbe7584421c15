// TMA descriptors of weight matrices (host side).
#pragma once
#include <cuda.h>
#include <string.h>

#include "common.cuh"

namespace ink {

typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// (driver entry point resolved at first use; no link to libcuda)
inline TensorMapEncodeFn tensor_map_encoder() {
  static TensorMapEncodeFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (TensorMapEncodeFn)p;
  }
  return fn;
}

// [columns] x rows x experts of one- or two-byte elements, box of box_columns x box_rows x 1 expert
inline int encode_rows(CUtensorMap* out, const void* base, int element_bytes, uint64_t expert_stride, int experts, int rows, int columns,
                       int box_columns, int box_rows, bool swizzle) {
  TensorMapEncodeFn enc = tensor_map_encoder();
  INK_REQUIRE(enc != nullptr, kLaunchFailed, "encode_rows: the driver has no cuTensorMapEncodeTiled");
  const uint64_t row_bytes = (uint64_t)columns * element_bytes;
  INK_REQUIRE(base != nullptr && aligned16(base) && expert_stride % 16 == 0 && expert_stride >= (uint64_t)rows * row_bytes,
              kBadArgument, "encode_rows: bank at %p with expert stride %llu", base, (unsigned long long)expert_stride);
  cuuint64_t dims[3] = {(cuuint64_t)columns, (cuuint64_t)rows, (cuuint64_t)experts};
  cuuint64_t strides[2] = {(cuuint64_t)row_bytes, (cuuint64_t)expert_stride};
  cuuint32_t box[3] = {(cuuint32_t)box_columns, (cuuint32_t)box_rows, 1}, elem[3] = {1, 1, 1};
  const CUresult r = enc(out, element_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(base), dims,
                         strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  INK_REQUIRE(r == CUDA_SUCCESS, kBadArgument, "encode_rows: cuTensorMapEncodeTiled returned %d", (int)r);
  return kOk;
}

}  // namespace ink
