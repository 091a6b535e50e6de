// The products of one fragment tile (qlayout.cuh: 16 weight rows x 128 k) with up to 8 NT activation rows on mma.sync.
#pragma once

#include "common.cuh"
#include "qlayout.cuh"

namespace tq {

// mma with a zero accumulator input (the compiler then needs no registers for it)
__device__ __forceinline__ void mma_bf16_16816_z(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                 uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// acc += the tile's products (FRESH: acc = them).  words(j, a): the integers of block j as bf16 pairs, a[row half][k pairs (0,1) (2,3) (4,5)
// (6,7) of this lane's eight]; rows(i, j): the same k of activation row 8 i + g; sc[row half][block]: the scales (not read for I8_ROW).
// mma.sync truncates when it adds to its accumulator, so only the two steps of a 32-block share one; the blocks of a tile are
// added in f32 first, and the tile's sum to acc: one accumulator over all of K had a bias of 2e-7 of the int8 results, the blocks
// added to acc one by one errors up to 1.25 times the general kernel's (24576 x 1536: 7.7e-8 there, 9.7e-8 one by one).
template <int KIND, int NT, bool FRESH = false, class Words, class Rows>
__device__ __forceinline__ void tile_sums(float (&acc)[NT][4], const float (&sc)[2][4], Words words, Rows rows) {
  float sum[NT][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t a[2][4];
    words(j, a);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const uint4 b = rows(i, j);
      float d[4];
      mma_bf16_16816_z(d, a[0][0], a[1][0], a[0][1], a[1][1], b.x, b.y);
      mma_bf16_16816(d, a[0][2], a[1][2], a[0][3], a[1][3], b.z, b.w);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if constexpr (KIND == I8_ROW) sum[i][c] = j == 0 ? d[c] : sum[i][c] + d[c];
        else sum[i][c] = j == 0 ? sc[c >> 1][j] * d[c] : fmaf(sc[c >> 1][j], d[c], sum[i][c]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = FRESH ? sum[i][c] : acc[i][c] + sum[i][c];
}

}  // namespace tq
