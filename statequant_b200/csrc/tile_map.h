// The tensor map of a state table's codes for the tensor-core kernels: [slot][row of the slot][bytes of a row], copied 128 rows
// at a time into a stage, 16-byte chunks swizzled (mma_pass.cuh).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>
#include "delta_step.cuh"
#include "fold_mma.cuh"

namespace sqb {

// What a tensor map takes of a table (codes of d_k 128): base and stride on 16 bytes, the stride positive and below 2^40.
inline bool tile_map_ok(const StepArgs& a) {
  return (reinterpret_cast<uintptr_t>(a.S) & 15) == 0 && a.sS > 0 && a.sS % 16 == 0 && a.sS < (1LL << 40);
}
// 0 or a CUDA error
inline int tile_map(TileMap& map, const StepArgs& a, int bits) {
  static_assert(sizeof(TileMap) == sizeof(CUtensorMap), "a TileMap holds a CUtensorMap");
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult got = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &got) != cudaSuccess || got != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Encode>(f);
  }();
  if (encode == nullptr) return static_cast<int>(cudaErrorNotSupported);
  const cuuint32_t rowb = 128 * bits / 8;
  // (the number of slots is the caller's affair: any int32 index)
  const cuuint64_t dims[3] = {rowb, static_cast<cuuint64_t>(a.HV) * a.DV, 2147483647ull}, strides[2] = {rowb, static_cast<cuuint64_t>(a.sS)};
  const cuuint32_t box[3] = {rowb, 128, 1}, one[3] = {1, 1, 1};
  CUtensorMap m;
  const CUresult r = encode(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, a.S, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            bits == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return static_cast<int>(cudaErrorInvalidValue);
  memcpy(map.bytes, &m, sizeof m);
  return 0;
}

}  // namespace sqb
