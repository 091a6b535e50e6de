// Host-side access to cuTensorMapEncodeTiled without linking libcuda.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace tq {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// (Asked for once, whichever host thread comes first; the others wait for the answer.)
inline EncodeTiledFn encode_tiled() {
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}

// bf16 matrix [rows][cols] with `ld` elements between rows, boxes of 64 columns x `box_rows` rows in the 128-byte
// swizzle; reads outside the matrix give zeros.  The base must be 16-byte aligned and ld a multiple of 8.
inline bool encode_bf16_k64(CUtensorMap* map, const void* base, size_t rows, size_t cols, size_t ld, unsigned box_rows) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t gstride[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstride, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same matrix, boxes of `box_blocks` neighbouring blocks of 64 columns, one behind the other in shared memory.  cols: a multiple of 64.
inline bool encode_bf16_k64_blocks(CUtensorMap* map, const void* base, size_t rows, size_t cols, size_t ld, unsigned box_rows, unsigned box_blocks) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t gdim[3] = {64, (cuuint64_t)rows, (cuuint64_t)(cols / 64)};
  const cuuint64_t gstride[2] = {(cuuint64_t)ld * 2, 128};
  const cuuint32_t box[3] = {64, box_rows, box_blocks};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), gdim, gstride, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Bytes [blocks][lines][128], boxes of `box_lines` lines of `box_blocks` blocks in the 128-byte swizzle (16-byte chunk c of line l
// of a 1024-byte aligned destination lands at chunk c ^ (l & 7)); lines behind a block's last read as zeros.
inline bool encode_lines128(CUtensorMap* map, const void* base, size_t lines, size_t blocks, unsigned box_lines, unsigned box_blocks) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t gdim[3] = {128, (cuuint64_t)lines, (cuuint64_t)blocks};
  const cuuint64_t gstride[2] = {128, (cuuint64_t)lines * 128};
  const cuuint32_t box[3] = {128, box_lines, box_blocks};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tq
