// Shared by the attention kernels that walk key tiles of 128 with tcgen05 (gqa_prefill_umma.cu, diff_attention_umma.cu).
#pragma once

#include "qgemm_umma.cuh"
#include "tensormap.h"

namespace tq {

constexpr int kPfTile = 128;                          // keys of a tile, rows of a query tile
constexpr int kPfBox = kPfTile * 128;                 // bytes of 128 rows of 64 bf16

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void pf_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
               "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
                 "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                 "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]) : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// Shared-memory descriptor of an operand whose rows are k and whose 64-element columns are contiguous (MN-major, 128-byte
// swizzle), in boxes of 128 k: the next 64 columns a box on, the next eight k 1024 bytes on.
__device__ __forceinline__ uint64_t pf_desc_mn(const void* smem_ptr) {
  return (uint64_t)((smem_u32(smem_ptr) >> 4) & 0x3FFF) | (uint64_t)(kPfBox >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

// One row's softmax attention over keys first .. end - 1, key by key in a warp: lane i has values KD i .. of the query and the keys, and 4 i .. of
// the 128 values' sums.  For the rows of a tile that met, with probability zero, an infinity or a NaN in the values of a key that they do not see: zero
// times that is NaN.  (Stops when every sum is NaN, as in a row that sees nothing else.)
template <int KD>
__device__ __forceinline__ void attend_row(const __nv_bfloat16* k, size_t k_ld, const __nv_bfloat16* v, size_t v_ld, int first, int end, const float (&q)[KD],
                                           float scale_log2, int lane, float& m, float& l, float (&acc)[4]) {
#pragma unroll 1
  for (int key = first; key < end; ++key) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < KD; ++i) s = fmaf(q[i], __bfloat162float(k[(size_t)key * k_ld + KD * lane + i]), s);
    s = warp_sum(s) * scale_log2;
    const float mn = fmaxf(m, s), f = ex2(m - mn), w = ex2(s - mn);
    m = mn;
    l = l * f + w;
    bool nan = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[i] = acc[i] * f + w * __bfloat162float(v[(size_t)key * v_ld + 4 * lane + i]);
      nan = nan && acc[i] != acc[i];
    }
    if (__all_sync(0xffffffffu, nan)) break;
  }
}

// bf16 [d2][d1][d0] with byte strides, boxes of 64 x b1 x b2 in the 128-byte swizzle; what lies outside reads as zeros.
inline bool encode_bf16_boxes(CUtensorMap* map, const void* base, size_t d0, size_t d1, size_t d2, size_t stride1, size_t stride2, unsigned b1, unsigned b2) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t gdim[3] = {d0, d1, d2}, gstride[2] = {stride1, stride2};
  const cuuint32_t box[3] = {64, b1, b2}, estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tq
