// Dequant-GEMM on the 5th-generation tensor cores (tcgen05 + tensor memory) for many activation
// rows (prefill, large decode batches, batched experts):
//     y[m, n] = sum_k x[m, k] * q[n, k] * scale[n, k/32]
// restating crates/tang-infer/src/quantize.rs:256-289 (q4_matvec, one call per activation row) as
// one contraction.
//
// Operand roles are swapped so that any token count fits one instruction shape: the 128 output
// features of a CTA are the UMMA M dimension (A operand, the dequantised weights), the tokens are
// the UMMA N dimension (B operand, 16..192), and the f32 accumulators D[128 x tokens] live in
// tensor memory.  Per chunk of 128 k:
//   * warp 0 streams the packed fragment tiles (tensor copies of 128-byte lines, swizzled so that the row-per-thread reads below
//     hit all banks), warp 2 the activations (boxes of 64 k, 128-byte swizzle, out-of-range token rows filled with zeros), each as
//     far ahead as its own ring allows;
//   * sixteen dequant warps, in two groups that each take every second chunk, turn the packed integers into bf16.  A thread owns one
//     output row = one tensor-memory lane and 64 k (a row's nibbles are 64 contiguous bytes of a tile) and writes them with
//     tcgen05.st.  The product q*scale (15 significant bits) is split into two bf16 numbers whose sum equals it EXACTLY, so two MMAs
//     per k-step reproduce exact products with f32 accumulation (TERMS = 2).  TERMS = 1 keeps the product
//     rounded to bf16 (relative weight error at most 2^-8), for bf16 outputs;
//   * one elected lane of warp 1 (even chunks) and of warp 3 (odd chunks) issues tcgen05.mma (kind::f16,
//     bf16 x bf16 -> f32; A from tensor memory), each into accumulators of its own, and commits each stage back to the producers;
//   * the dequant warps finally read the accumulators with tcgen05.ld, add them and store y.
// What bounds it, found with cycle counters: up to 64 rows first the threads that issue (a tensor copy 330 to 450 cycles with its wait and
// its announcement; an MMA issuer's turn 700 beside the MMAs), hence copies of 256 k of activations and turns of 128 k; then the
// conversion (1200 cycles of a group's 1640 per chunk, ALU and FMA pipes 60 % busy).  us per launch, chunks of 64 k -> as it is:
// 28672 x 4096 at 64 rows 42.0 -> 34.7, 4096 x 14336 22.8 -> 20.4, int8 7168 x 16384 44.7 -> 35.7, 1024 x 4096 at 1024 rows 19.7 -> 16.3.
// Every mbarrier wait is bounded; on failure the CTA records a code, skips ahead and still frees its
// tensor memory.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "qlayout.cuh"

namespace tq {

constexpr int kUmmaRows = 128;        // output features per CTA
constexpr int kUmmaK = 64;            // k of an activation box (one 128-byte swizzle span of bf16)
constexpr int kUmmaGroups = 2;        // dequant groups, each converting every second 128-k chunk
constexpr int kUmmaGroupWarps = 8;    // warps per group
constexpr int kUmmaDqWarps = kUmmaGroups * kUmmaGroupWarps;   // dequant / epilogue warps
constexpr int kUmmaFirstDqWarp = 4;   // warps 0..3: weight producer, MMA issuer (even steps), activation producer, MMA issuer (odd steps)
constexpr int kUmmaDualAcc = 96;      // two token tiles per CTA: columns between a tile's accumulators, where it has two
constexpr int kUmmaThreads = 32 * (kUmmaFirstDqWarp + kUmmaDqWarps);

struct UmmaParams {
  const float* row_scales;   // TQ_I8_ROW: one scale per output row (applied to the accumulator), else unused
  void* y;                // [M][ldy] f32 or bf16
  long long ldy;
  int m_total;            // activation rows
  int n_rows;             // output features (multiple of 128)
  int kc_total;           // K / 128
  int ntok;               // tokens per CTA tile = UMMA N (multiple of 16, <= 192)
  int acc_stride;         // columns between accumulators (two token tiles: between the tiles')
  int a_col0;             // tensor-memory columns of the converted weights: stages x 2 x terms x 32 from here on
  int n_acc;              // accumulators (2, 4 or 8): 64-k step j of issuer i adds into number i + 2 * (j % (n_acc / 2)) (two token tiles: see the kernel)
  int stages;             // stages of converted weights in tensor memory (128 k each; even)
  int x_slots, kx;        // slots of activations in shared memory, 64-k boxes per slot (4; more than 64 tokens 2, two token tiles 1)
  int raw_stages;         // packed-tile ring depth (slots of kt tiles of 128 k): what keeps the HBM stream in flight
  int kt;                 // k-tiles per ring slot (2 or 4)
  int y_bf16;
  int swiglu;             // 1: the weight is a gate/up projection in the interleaved row order (rows 0..7 of every 16 gate, rows
                          // 8..15 the matching up rows); 2: gate rows in the first half of the weight's (group's) rows, up rows in
                          // the second (no K split).  y [M][n_rows / 2] = silu(gate) * up, formed from the f32 sums
  int splits;             // CTAs along K per output tile (gridDim.z): a cluster
  int kc_per_split;       // 128-k tiles per split
  int run_kc;             // chunks that the accumulators sum before they are added up and start anew (even; 0: all)
  int y_vec4;             // four values of a row of y are stored at once
  const int* g_counts;    // grouped launches (experts stacked by rows): rows of x / y per group, or null
  const int* g_offsets;   // first row of each group
  int n_groups;
  int* err;
};

// Host-side description of a grouped launch (device arrays come from the router's bookkeeping kernels).
struct UmmaGroups {
  int n_groups = 1;
  const int* counts = nullptr;
  const int* offsets = nullptr;
  int max_active = 0;      // upper bound of groups with rows
  int expected_rows = 0;   // typical counts[e]: sets the token tile
};

__host__ __device__ inline size_t umma_box_bytes(int ntok) { return (size_t)ntok * 128; }   // 64 k of a token tile's activations
constexpr int kUmmaMaxRawStages = 16, kUmmaMaxStages = 4, kUmmaMaxXSlots = 4, kUmmaMaxSplits = 8;
constexpr int kUmmaHeader = 1024;
__host__ __device__ inline size_t umma_smem_bytes(int kind, size_t x_ring, int raw_tiles) {
  return kUmmaHeader + 1024 /*alignment slack*/ + x_ring +
         (size_t)raw_tiles * 8 * qk_tile_bytes(kind);
}

// ---- PTX wrappers -------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* slot_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Sixteen 32-bit columns of the calling warp's 32 lanes: thread i writes lane i (registers = consecutive columns).
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) { asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory"); }

// D[tmem] (+)= A[tmem] * B[smem descriptor]: the A operand is read from tensor memory (lane = row, each 32-bit
// column holds two consecutive k as bf16, eight columns per 16-k instruction).
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(const void* smem_ptr) {
  const uint32_t addr = smem_u32(smem_ptr);
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);        // start address, 16-byte units
  d |= (uint64_t)1 << 16;                       // leading byte offset (unused with swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;             // stride byte offset: next 8-row group
  d |= (uint64_t)1 << 46;                       // descriptor version of this architecture
  d |= (uint64_t)2 << 61;                       // 128-byte swizzle
  return d;
}

// Instruction descriptor, kind::f16: D f32, A bf16, B bf16, both K-major, M = 128, N = ntok.
// (A and B must have the same format: an f16 A with a bf16 B is rejected by the hardware as an
// illegal instruction.)
__host__ __device__ inline uint32_t umma_idesc_bf16(int ntok) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ntok >> 3) << 17) | ((uint32_t)(kUmmaRows >> 4) << 24);
}

}  // namespace tq
