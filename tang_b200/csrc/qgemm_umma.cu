// tcgen05 / tensor-memory dequant-GEMM: kernel and launcher (see qgemm_umma.cuh for the design).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "internal.h"
#include "qgemm_umma.cuh"
#include "tensormap.h"

namespace tq {

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The sum of the four floats at `mine` over the first n CTAs of the cluster, in their order.
__device__ __forceinline__ float4 cluster_sum(const float* mine, int n) {
  const uint32_t a = smem_u32(mine);
  float4 v[kUmmaMaxSplits];
#pragma unroll
  for (int z = 0; z < kUmmaMaxSplits; ++z) {
    if (z >= n) break;
    uint32_t there;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(a), "r"(z));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[z].x), "=f"(v[z].y), "=f"(v[z].z), "=f"(v[z].w) : "r"(there) : "memory");
  }
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int z = 0; z < kUmmaMaxSplits; ++z) {
    if (z >= n) break;
    sum.x += v[z].x;
    sum.y += v[z].y;
    sum.z += v[z].z;
    sum.w += v[z].w;
  }
  return sum;
}
__device__ __forceinline__ float4 times(float4 v, const float* s) { return make_float4(v.x * s[0], v.y * s[1], v.z * s[2], v.w * s[3]); }

// Adds the accumulators' columns c0 .. c0 + 15 of this warp's lanes up, in their order: number a is issuer a & 1's, which has reached it if it had
// more than a >> 1 steps (steps0, steps1).
__device__ __forceinline__ void sum_accumulators(uint32_t tmem_lanes, const UmmaParams& p, int c0, int steps0, int steps1, float (&v)[16]) {
  float u[16];
  tmem_ld16(tmem_lanes + (uint32_t)c0, v);
  for (int a = 1; a < p.n_acc; ++a) {
    if ((a >> 1) >= ((a & 1) ? steps1 : steps0)) continue;
    tmem_ld16(tmem_lanes + (uint32_t)(a * p.acc_stride + c0), u);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += u[i];
  }
}

template <int KIND, int TERMS, int DUAL = 0, bool RUNS = false>
__global__ void __launch_bounds__(kUmmaThreads, 1)
qgemm_umma_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ UmmaParams p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int TB = (KIND == I8_ROW) ? 2048 : (KIND == Q8_F32) ? 2304 : (KIND == Q4_F16) ? 1152 : 1280;
  constexpr bool kIs8 = KIND == I8_ROW || KIND == Q8_F32;
  constexpr bool kExactSplit = KIND == Q4_F16 && TERMS == 2;
  constexpr int kTileLines = TB / 128;   // 128-byte lines of a tile: its weights, then its scales
  static_assert(KIND != I8_ROW || TERMS == 1, "int8 rows carry no scale into the operand: one exact term");
  // DUAL: the CTA covers two token tiles of p.ntok rows with one conversion of the weights: issuer warp 1 multiplies
  // every stage with the first tile's activations, warp 3 with the second tile's, each into DUAL accumulators
  static_assert(!DUAL || TERMS == 1, "two token tiles per CTA: single-term weights");
  // RUNS: the sums are cut every p.run_kc chunks: the epilogue's warps add the accumulators up in f32, in shared memory of their own (registers
  // held over the conversion cost it a tenth), and the issuers start them anew.
  static_assert(!DUAL || !RUNS, "cut sums: one token tile per CTA");
  constexpr int kTokTiles = DUAL ? 2 : 1;
  // ---- shared-memory carve-up (operand tiles need 1024-byte alignment for the 128-byte swizzle)
  uint8_t* smem = smem_raw;
  uint64_t* x_full = reinterpret_cast<uint64_t*>(smem);       // [x slots] activation boxes landed
  uint64_t* x_empty = x_full + kUmmaMaxXSlots;                 // [x slots] MMAs that read them retired (one commit per issuer that does)
  uint64_t* a_full = x_empty + kUmmaMaxXSlots;                 // [stages] weights written (one arrival per dequant warp)
  uint64_t* empty = a_full + kUmmaMaxStages;                   // [stages] MMAs of the stage retired (two token tiles: x_empty of its second box)
  uint64_t* raw_full = empty + kUmmaMaxStages;                 // [raw stages] packed tiles landed
  uint64_t* raw_empty = raw_full + kUmmaMaxRawStages;             // [raw stages] packed tiles consumed (one arrival per dequant warp)
  uint64_t* acc_full = raw_empty + kUmmaMaxRawStages;             // accumulator complete
  uint64_t* acc_free = acc_full + 1;                           // accumulators of a run read (RUNS)
  uint64_t* x_tail = acc_free + 1;                             // a last chunk that both issuers share: its activations landed,
  uint64_t* a_tail = x_tail + 1;                               // its weights written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(a_tail + 1);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t base_u32 = smem_u32(smem_raw);
  uint8_t* tiles_s = smem_raw + kUmmaHeader + ((1024 - ((base_u32 + kUmmaHeader) & 1023)) & 1023);  // 1024-aligned
  const int KX = DUAL ? 1 : p.kx;                              // 64-k steps per activation slot
  const size_t x_bytes = umma_box_bytes(p.ntok) * kTokTiles * KX;
  float* part_s = reinterpret_cast<float*>(tiles_s);            // K split: this CTA's partial sums, when the rings are done with
  uint8_t* raw_s = tiles_s + (size_t)p.x_slots * x_bytes;   // [raw stages][8 tiles]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.stages, XS = p.x_slots, RS = p.raw_stages, KT = p.kt;
  // The eight 16-row blocks of this CTA come in two boxes of four: neighbours, or (swiglu 2) gate blocks and their up blocks
  int rb_first = (int)blockIdx.x * (p.swiglu == 2 ? 4 : 8);
  const int rb_away = p.swiglu == 2 ? p.n_rows / (2 * kTileRows) : 4;
  int m0 = blockIdx.y * p.ntok * kTokTiles;                    // first token of this CTA
  int m_end = p.m_total;                                       // rows at or beyond this are not this CTA's to store
  const float* row_scales = p.row_scales;   // TQ_I8_ROW: per output row, applied to the accumulator
  int ntok = p.ntok;                                           // tokens of this CTA's tile: the MMA's N
  if (p.g_counts) {
    // Grouped (experts): the token tiles of all groups are numbered one group after the other, and blockIdx.y is such a number (the grid
    // has as many as there can be; a place per group and possible tile, most of them empty, cost 64 experts at 4096 tokens
    // 40,000 CTAs that left at once).  Group e's rows are g_offsets[e] .. +g_counts[e] of x and y, evened out over its tiles, its weights
    // n_rows further on.
    pdl_wait();
    int* mine = reinterpret_cast<int*>(smem_raw + kUmmaHeader) - 3;   // (the header's end; a static array would not fit beside the rings)
    if (warp == 0) {
      int before = 0, e = -1, tile = 0, tiles = 1;
      for (int g0 = 0; g0 < p.n_groups && e < 0; g0 += 32) {
        const int n = g0 + lane < p.n_groups ? (p.g_counts[g0 + lane] + p.ntok - 1) / p.ntok : 0;
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += u;
        }
        const unsigned behind = __ballot_sync(0xffffffffu, before + upto > (int)blockIdx.y);
        if (behind) {
          const int l = __ffs(behind) - 1;
          e = g0 + l;
          tiles = __shfl_sync(0xffffffffu, n, l);
          tile = (int)blockIdx.y - (before + __shfl_sync(0xffffffffu, upto, l) - tiles);
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
      }
      if (lane == 0) {
        mine[0] = e;
        mine[1] = tile;
        mine[2] = tiles;
      }
    }
    __syncthreads();
    const int e = mine[0];
    if (e < 0) return;
    const int cnt = p.g_counts[e];
    ntok = ((cnt + mine[2] - 1) / mine[2] + 15) & ~15;
    m0 = p.g_offsets[e] + mine[1] * ntok;
    m_end = p.g_offsets[e] + cnt;
    rb_first += e * (p.n_rows / kTileRows);
    row_scales += (size_t)e * p.n_rows;
  }
  const int kc_begin = p.g_counts ? 0 : blockIdx.z * p.kc_per_split;   // this CTA's slice of K, in 128-k tiles
  const int kc_len = min(p.kc_per_split, p.kc_total - kc_begin);
  // An odd number of chunks with one accumulator per issuer: the issuers take half of the last chunk each, so that both accumulators see as
  // many additions (K = 128 at 65 rows and more, int4: error 1.9e-7 otherwise, 1.2e-7 so).  That chunk has barriers of its own, used once: a wait for
  // a parity is not sound in an issuer that has not seen the stage's phases before.  (Weights rounded to bf16 have no use for it.)
  constexpr bool kTail = !DUAL && (TERMS == 2 || KIND == I8_ROW);
  const bool shared_tail = kTail && p.n_acc == 2 && (kc_len & 1);

  if (warp == 0) {
    if (lane < XS) {
      mbar_init(&x_full[lane], 1);
      mbar_init(&x_empty[lane], p.kx == 2 ? 1 : 2);
    }
    if (lane < S) {
      mbar_init(&a_full[lane], kUmmaGroupWarps);
      mbar_init(&empty[lane], 1);
    }
    if (lane < RS) {
      mbar_init(&raw_full[lane], 1);
      mbar_init(&raw_empty[lane], kUmmaDqWarps);          // every group reads some tile of every ring slot
    }
    if (lane == 0) {
      mbar_init(acc_full, 2);
      if (RUNS) mbar_init(acc_free, kUmmaDqWarps);
      if (kTail) {
        mbar_init(x_tail, 1);
        mbar_init(a_tail, kUmmaGroupWarps);
      }
      *failed = 0;
    }
    mbar_init_fence();
  } else if (warp == 2 && lane == 0) {
    prefetch_map(&x_map);
    prefetch_map(&w_map);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = *tmem_slot;

  // (weights are not written by a kernel in flight -- their constructors end with a launch or a wait that sees to it --: they stream and are
  // converted before the wait for the activations, which the thread that copies them does; everything that is stored depends on these)
  pdl_launch_dependents();

  auto give_up = [&](int code) {
    *failed = 1;
    atomicCAS(p.err, 0, code);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ packed-weight producer
    if (lane == 0) {
      const uint64_t pol_w = l2_policy_evict_first();
      int r = 0;
      uint32_t rph = 0;
      // one ring slot = KT consecutive k-tiles of the CTA's eight row blocks, in two boxes of 128-byte lines (tiles behind
      // the matrix's last read as zeros and are not looked at)
      for (int t0 = 0; t0 < kc_len && !*failed; t0 += KT) {
        if (!mbar_wait_spin(&raw_empty[r], rph ^ 1u)) { give_up(DERR_EMPTY_WAIT); break; }
        mbar_arrive_expect_tx(&raw_full[r], 8u * KT * TB);
        uint8_t* slot = raw_s + (size_t)r * 8 * KT * TB;
        tma_load_3d(slot, &w_map, 0, (kc_begin + t0) * kTileLines, rb_first, &raw_full[r], pol_w);
        tma_load_3d(slot + 4 * KT * TB, &w_map, 0, (kc_begin + t0) * kTileLines, rb_first + rb_away, &raw_full[r], pol_w);
        if (++r == RS) {
          r = 0;
          rph ^= 1u;
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ activation producer
    // Waiting for a slot, announcing the bytes and issuing one copy takes this thread 330 to 450 cycles, which is more than a step of
    // few tokens: a copy brings KX boxes of 64 k.
    if (lane == 0) {
      pdl_wait();
      int s = 0;
      uint32_t ph = 0, tok = 1;
      for (int kb = 0; kb < 2 * (kc_len - shared_tail); kb += KX) {
        if (!mbar_wait_token(&x_empty[s], ph ^ 1u, tok)) { give_up(DERR_EMPTY_WAIT); break; }
        mbar_arrive_expect_tx(&x_full[s], (uint32_t)(p.ntok * kTokTiles * KX) * 128u);
        uint8_t* slot = tiles_s + (size_t)s * x_bytes;
        // (rows and k beyond the matrix read as zeros, a box entirely beyond it too)
        tma_load_3d(slot, &x_map, 0, m0, kc_begin * 2 + kb, &x_full[s]);
        if constexpr (DUAL) tma_load_3d(slot + (size_t)p.ntok * 128, &x_map, 0, m0 + p.ntok, kc_begin * 2 + kb, &x_full[s]);
        if (++s == XS) {
          s = 0;
          ph ^= 1u;
          if (*failed) break;
        }
        tok = mbar_test(&x_empty[s], ph ^ 1u);
      }
      if (shared_tail && !*failed) {
        if (mbar_wait_token(&x_empty[s], ph ^ 1u, tok)) {
          mbar_arrive_expect_tx(x_tail, (uint32_t)(p.ntok * 2) * 128u);
          tma_load_3d(tiles_s + (size_t)s * x_bytes, &x_map, 0, m0, 2 * (kc_begin + kc_len - 1), x_tail);
        } else {
          give_up(DERR_EMPTY_WAIT);
        }
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ------------------------------------------------------------------ MMA issuers
    // Two of them: a chunk of 128 k takes an issuer's thread its MMAs (~45 cycles each) and several hundred cycles for waits and
    // commits, so warp 1 takes the even chunks into the even accumulators and warp 3 the odd chunks into the odd ones; the
    // epilogue adds them all (a fixed order: reproducible).  With even rings an issuer returns to stages that it consumed itself.
    // The whole warp runs the loop (warp-uniform control flow keeps the descriptors in uniform registers); one elected lane issues.
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc_bf16(ntok);
    const int odd = warp == 3;
    const uint32_t box_u = (uint32_t)((p.ntok * 128) >> 4), slot_u = (uint32_t)(x_bytes >> 4);
    // slots of four boxes serve a chunk of either issuer, slots of two one chunk; with two token tiles (a box of each per slot) a
    // chunk takes two slots and every issuer every chunk
    const uint64_t desc0 = umma_desc_sw128(tiles_s) + (DUAL ? (uint32_t)odd * box_u : KX == 4 ? 2u * odd * box_u : 0u);
    const uint32_t half_u = DUAL ? slot_u : box_u;
    // Each issuer rotates over n_acc / 2 accumulators: the tensor core truncates every f32 addition, an error that
    // grows with the number of additions one accumulator sees, so as many short sums as tensor memory holds
    // (512 columns) are kept and the epilogue adds them, in accumulator order.
    const int rot_mask = (p.n_acc >> 1) - 1;
    int j = 0;                                  // this issuer's 64-k steps
    constexpr int kStep = DUAL ? 1 : 2;
    const int x_step = KX == 4 ? 1 : 2;
    int s = DUAL ? 0 : odd, xs = DUAL || KX == 4 ? 0 : odd;     // stage of weights; activation slot
    uint32_t ph = 0, xph = 0, tok_a = 0;
    bool ok = true;
    int ck = DUAL ? 0 : odd, run = 0;
    // (run_kc is even: every run but the last has as many chunks for either issuer)
    for (int run_end = RUNS ? min(p.run_kc, kc_len) : kc_len;; run_end = min(run_end + p.run_kc, kc_len), ++run) {
      const int ck_end = run_end == kc_len ? kc_len - shared_tail : run_end;
      j = 0;
#pragma unroll 1
      for (; ck < ck_end; ck += kStep) {
        ok = mbar_wait_token(&a_full[s], ph, tok_a) && mbar_wait_spin(&x_full[xs], xph);
        if (!ok) { give_up(DERR_FULL_WAIT); break; }
        tc_fence_after();
        const uint64_t xd = desc0 + (uint64_t)((uint32_t)xs * slot_u);
        const uint32_t a_t0 = tmem_d + (uint32_t)(p.a_col0 + s * (64 * TERMS));
#pragma unroll
        for (int half = 0; half < 2; ++half, ++j) {
          if (DUAL && half == 1) {
            ok = mbar_wait_spin(&x_full[xs + 1], xph);
            if (!ok) { give_up(DERR_FULL_WAIT); break; }
          }
          const uint32_t acc = tmem_d + (uint32_t)((DUAL ? odd : odd + 2 * (j & rot_mask)) * p.acc_stride) + (DUAL == 2 ? (uint32_t)(half * kUmmaDualAcc) : 0u);
          const uint32_t fresh = (DUAL ? j < DUAL : j <= rot_mask) ? 0u : 1u;   // the accumulator's first step overwrites it
          if (leader) {
#pragma unroll
            for (int k16 = 0; k16 < kUmmaK / 16; ++k16) {
              const uint64_t bd = xd + half * half_u + 2 * k16;
              // 32 columns (64 k) of the hi term, then 32 of the lo term
              const uint32_t a_t = a_t0 + (uint32_t)(half * (32 * TERMS) + 8 * k16);
              umma_f16_ts(acc, a_t, bd, idesc, fresh | (k16 != 0));
              if (TERMS == 2) umma_f16_ts(acc, a_t + 32u, bd, idesc, 1u);
            }
            // (commits arrive when the MMAs so far have finished reading)
            if (DUAL) umma_commit(&x_empty[xs + half]);
          }
        }
        if (!ok) break;
        if (!DUAL && leader) {
          umma_commit(&empty[s]);
          umma_commit(&x_empty[xs]);
        }
        __syncwarp();
        xs += x_step;
        if (xs >= XS) {
          xs -= XS;
          xph ^= 1u;
        }
        s += kStep;
        if (s >= S) {
          s -= S;
          ph ^= 1u;
        }
        // Look at the next chunk's barrier only now: the answer takes ~70 cycles, during which an in-order
        // thread issues nothing, and here the tensor core already has this chunk's work.
        tok_a = mbar_test(&a_full[s], ph);
      }
      if (!RUNS || run_end == kc_len || !ok) break;
      // the run's sums are complete when its products are, and the accumulators the next run's when they have been read
      if (leader) umma_commit(acc_full);
      __syncwarp();
      ok = mbar_wait_spin(acc_free, run & 1);
      if (!ok) {
        give_up(DERR_TMEM);
        break;
      }
      tc_fence_after();
    }
    if (shared_tail && ok) {                     // (slots of two boxes: a chunk each)
      ok = mbar_wait_spin(a_tail, 0) && mbar_wait_spin(x_tail, 0);
      if (!ok) give_up(DERR_FULL_WAIT);
      tc_fence_after();
      if (ok && leader) {
        const uint64_t xd = desc0 + (uint64_t)((uint32_t)((kc_len - 1) % XS) * slot_u + (uint32_t)odd * box_u);
        const uint32_t acc = tmem_d + (uint32_t)(odd * p.acc_stride);
        const uint32_t a_t0 = tmem_d + (uint32_t)(p.a_col0 + (kc_len - 1) % S * (64 * TERMS) + odd * (32 * TERMS));
#pragma unroll
        for (int k16 = 0; k16 < kUmmaK / 16; ++k16) {
          umma_f16_ts(acc, a_t0 + 8u * k16, xd + 2 * k16, idesc, (j | k16) != 0);
          if (TERMS == 2) umma_f16_ts(acc, a_t0 + 8u * k16 + 32u, xd + 2 * k16, idesc, 1u);
        }
      }
      __syncwarp();
    }
    if (leader) umma_commit(acc_full);           // arrives when every MMA issued so far has completed
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ dequant warps
    // Two groups of eight warps convert every second chunk of 128 k, four warps of a group (one per lane quarter of tensor memory) its
    // first 64 k, four the second: one chunk's chain of waits, loads, arithmetic, stores and fence is long, and the groups overlap it.
    const int group = (warp - kUmmaFirstDqWarp) / kUmmaGroupWarps;
    // This thread owns output row 32 * (warp % 4) + lane, i.e. that lane of tensor memory: row g + 8 h of tile rbi of the slot.  In
    // a tile the row's nibbles are 64 contiguous bytes (its four k quarters of 16 bytes, each holding one word per 32-block), its
    // scales 8 or 16 contiguous bytes.  The copy swizzles: bits 7..9 of a byte's place in the slot are added (xor) to
    // bits 4..6, so that the eight rows that a quarter warp reads, 64 bytes apart, lie in all 32 banks instead of in eight.
    const int q4 = warp & 3;
    const int rbi = p.swiglu == 2 ? (lane >> 4) * 4 + q4 : 2 * q4 + (lane >> 4), h = (lane >> 3) & 1, g = lane & 7;
    bool ok = true;
    const int c = ((warp - kUmmaFirstDqWarp) >> 2) & 1;          // which 64-k half of the chunk
    int s = group, r = 0, within = group;                        // stage; packed-tile slot and the tile inside it (KT is 2 or 4)
    uint32_t ph = 0, rph = 0;
    uint64_t* const stage_empty = DUAL ? x_empty + 1 : empty;
    constexpr int kEmptyStep = DUAL ? 2 : 1;
    uint32_t tok_raw = 0, tok_empty = 1;                         // (what is free is free at first)
    const uint32_t tmem_lanes = tmem_d + ((uint32_t)(32 * q4) << 16);
    const int col0 = 16 * ((warp - kUmmaFirstDqWarp) >> 2);      // four warps share a lane quarter and alternate over the 16-column chunks
    constexpr int kColStep = 16 * (kUmmaDqWarps / 4);
    float* const sums = reinterpret_cast<float*>(raw_s + (size_t)RS * 8 * KT * TB) + 32 * q4 + lane;   // RUNS: the runs so far, [token][128 features]
    int run = 0;
    int ck = group;
    // RUNS: the first group takes a run behind its first chunk of the next one, while the run's last products go on, the second, which converted the
    // run's last chunk, at once
    for (int stop = RUNS ? min(p.run_kc + (group ? 0 : kUmmaGroups), kc_len) : kc_len;; stop = min(stop + p.run_kc, kc_len)) {
      const int from = ck;
#pragma unroll 1
      for (; ck < stop; ck += kUmmaGroups) {
        // (with two terms the stage is only waited for when the first half of the row is converted:
        // the MMAs that last read it have that long to finish -- decode step at batch 64 8.27 -> 8.11 ms; with one term
        // the conversion is too short for that and the early wait measured 3 % better)
        constexpr bool kLateWait = TERMS == 2;
        ok = mbar_wait_token(&raw_full[r], rph, tok_raw) && (kLateWait || mbar_wait_token(&stage_empty[s * kEmptyStep], ph ^ 1u, tok_empty));
        if (!ok) { give_up(DERR_FULL_WAIT); break; }
        const int s_cur = s, r_cur = r, within_cur = within;
        const uint32_t ph_cur = ph;
        s += kUmmaGroups;
        if (s >= S) {
          s -= S;
          ph ^= 1u;
        }
        within += kUmmaGroups;
        const bool leaves = within >= KT;           // this group's next tile lies in the next ring slot
        if (leaves) {
          within -= KT;
          if (++r == RS) {
            r = 0;
            rph ^= 1u;
          }
        }
        const uint8_t* slot = raw_s + (size_t)r_cur * 8 * KT * TB;
        const int tile_line = (rbi * KT + within_cur) * kTileLines;      // the tile's first line in the slot
        if (!kLateWait) tc_fence_after();          // the stage's columns were last read by MMAs whose commit was waited for
        const int line = tile_line + (kIs8 ? 8 * h + 4 * c : 4 * h) + (g >> 1);
        const uint8_t* wrow = slot + line * 128 + (kIs8 ? 0 : 8 * c);
        const int chunk0 = ((g & 1) * 4) ^ (line & 7);
        const uint32_t a_t = tmem_d + ((uint32_t)(32 * q4) << 16) + (uint32_t)(p.a_col0 + s_cur * (64 * TERMS) + c * (32 * TERMS));
        uint32_t sh = 0, sl = 0;
        if constexpr (KIND != I8_ROW) {
          // Two terms of Q4 with f16 scales: s_hi = the scale rounded to five significant bits and s_lo = the rest, which has
          // five too (of 11, rounded to nearest).  The integers have three (or are -8), so both products are exact in bf16, and
          // so is 24 * s: each term is one fma over 24 + q, half the instructions of the general form below.
          // General form: the scale as s_hi + s_lo, two bf16 numbers (exact for an f16 scale: 11 = 8 + 3 significant bits).
          // With t = q*s_lo (7 bits, exact in bf16), hi = fma(q, s_hi, t) is the exact product rounded once;
          // lo = t - fma(q, -s_hi, hi) = q*scale - hi, both steps exact, so hi + lo reproduces the product.
          // (f32 scales keep their first 16 significant bits this way, and with int8 values t itself is rounded to 8
          // bits: hi + lo is then the product to within 2^-15 relative.)
          float2 f;
          const int s_line = tile_line + (kIs8 ? 16 : 8) + (KIND == Q4_F16 ? 0 : h);
          if (KIND == Q4_F16) f = __half22float2(*reinterpret_cast<const __half2*>(slot + s_line * 128 + (((4 * h + (g >> 1)) ^ (s_line & 7)) << 4) + 8 * (g & 1) + 4 * c));
          else f = *reinterpret_cast<const float2*>(slot + s_line * 128 + ((g ^ (s_line & 7)) << 4) + 8 * c);
          if constexpr (kExactSplit) {
            const uint32_t h0 = (__float_as_uint(f.x) + 0x40000u) & 0xFFF80000u, h1 = (__float_as_uint(f.y) + 0x40000u) & 0xFFF80000u;
            sh = prmt(h0, h1, 0x7632u);
            sl = prmt(__float_as_uint(f.x - __uint_as_float(h0)), __float_as_uint(f.y - __uint_as_float(h1)), 0x7632u);
          } else {
          const __nv_bfloat162 shb = __floats2bfloat162_rn(f.x, f.y);
          sh = *reinterpret_cast<const uint32_t*>(&shb);
          const __nv_bfloat162 slb = __floats2bfloat162_rn(f.x - __uint_as_float(sh << 16), f.y - __uint_as_float(sh & 0xFFFF0000u));
          sl = *reinterpret_cast<const uint32_t*>(&slb);
          }
        }
        uint32_t wq[4][4];                         // [k quarter][word]: Q4 uses words 0, 1 (blocks 2c, 2c+1)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if constexpr (kIs8) {
            const uint4 v = *reinterpret_cast<const uint4*>(wrow + ((chunk0 ^ t) << 4));
            wq[t][0] = v.x; wq[t][1] = v.y; wq[t][2] = v.z; wq[t][3] = v.w;
          } else {
            const uint2 v = *reinterpret_cast<const uint2*>(wrow + ((chunk0 ^ t) << 4));
            wq[t][0] = v.x; wq[t][1] = v.y; wq[t][2] = 0u; wq[t][3] = 0u;
          }
        }
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          uint32_t hi[16], lo[16];
          if constexpr (kExactSplit) {
            const uint32_t s_hi = prmt(sh, sh, jj ? 0x3232u : 0x1010u), s_lo = prmt(sl, sl, jj ? 0x3232u : 0x1010u);
            const uint32_t c_hi = bf16x2_mul(s_hi, 0xC1C0C1C0u), c_lo = bf16x2_mul(s_lo, 0xC1C0C1C0u);   // -24 s
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              uint32_t v[4];                         // 24 + q of (k0,k1) (k2,k3) (k4,k5) (k6,k7) of k quarter t
              dequant_q4_word_24(wq[t][jj], v);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                hi[4 * t + e] = bf16x2_fma(v[e], s_hi, c_hi);
                lo[4 * t + e] = bf16x2_fma(v[e], s_lo, c_lo);
              }
            }
          } else {
          const uint32_t s_hi = prmt(sh, sh, jj ? 0x3232u : 0x1010u), s_lo = prmt(sl, sl, jj ? 0x3232u : 0x1010u), minus_s_hi = s_hi ^ 0x80008000u;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            uint32_t q[4];                         // (k0,k1) (k2,k3) (k4,k5) (k6,k7) of k quarter t, exact ints
            if constexpr (kIs8) dequant_i8_words(wq[t][2 * jj], wq[t][2 * jj + 1], q);
            else dequant_q4_word(wq[t][jj], q);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if constexpr (KIND == I8_ROW) {
                hi[4 * t + e] = q[e];
              } else {
                const uint32_t tt = bf16x2_mul(q[e], s_lo);
                hi[4 * t + e] = bf16x2_fma(q[e], s_hi, tt);
                if (TERMS == 2) lo[4 * t + e] = bf16x2_sub(tt, bf16x2_fma(q[e], minus_s_hi, hi[4 * t + e]));
              }
            }
          }
          }
          if (kLateWait && jj == 0) {
            // the stage's columns were last read by MMAs whose commit is waited for here
            ok = __all_sync(0xffffffffu, mbar_wait_token(&stage_empty[s_cur * kEmptyStep], ph_cur ^ 1u, tok_empty));
            tc_fence_after();
          }
          if (ok) {
            tmem_st16(a_t + (uint32_t)(16 * jj), hi);
            if (TERMS == 2) tmem_st16(a_t + (uint32_t)(32 + 16 * jj), lo);
          }
        }
        if (!ok) { give_up(DERR_EMPTY_WAIT); break; }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {                                                // one arrival per warp
          mbar_arrive(&a_full[s_cur]);
          if (leaves) mbar_arrive(&raw_empty[r_cur]);   // done with this ring slot (nobody waits for the final ones)
        }
        if (ck + kUmmaGroups < kc_len) {               // early look at what this group's next stage waits for
          tok_raw = leaves ? mbar_test(&raw_full[r], rph) : 1u;
          tok_empty = mbar_test(&stage_empty[s * kEmptyStep], ph ^ 1u);
        }
      }
      if (shared_tail && stop == kc_len && from < kc_len && group == 0 && lane == 0) mbar_arrive(a_tail);   // (the last chunk was this group's)
      if (!RUNS || !ok || (run + 1) * p.run_kc >= kc_len) break;
      ok = __all_sync(0xffffffffu, mbar_wait_spin(acc_full, run & 1));
      if (!ok) break;
      tc_fence_after();
      for (int c0 = col0; c0 < ntok; c0 += kColStep) {
        float v[16];
        sum_accumulators(tmem_lanes, p, c0, p.run_kc, p.run_kc, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) sums[(c0 + i) * kUmmaRows] = run ? sums[(c0 + i) * kUmmaRows] + v[i] : v[i];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
      ++run;
    }
    // ---- epilogue: D[128 features x ntok tokens] -> y[token][feature]
    if (ok && !*failed) ok = mbar_wait_spin(acc_full, run & 1);
    if (!ok) give_up(DERR_TMEM);
    tc_fence_after();
    if (ok) {
      const int n = blockIdx.x * kUmmaRows + 32 * q4 + lane;
      const int kc_run = RUNS ? kc_len - run * p.run_kc : kc_len;
      for (int tile = 0; tile < kTokTiles; ++tile)
      for (int c0 = col0; c0 < ntok; c0 += kColStep) {
        float v[16];
        const int mt = m0 + tile * p.ntok;                // first token of the tile
        if constexpr (DUAL) {
          float v1[16];
          tmem_ld16(tmem_lanes + (uint32_t)(tile * p.acc_stride + c0), v);
          if (DUAL == 2) {
            tmem_ld16(tmem_lanes + (uint32_t)(tile * p.acc_stride + kUmmaDualAcc + c0), v1);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += v1[i];
          }
        } else {
          sum_accumulators(tmem_lanes, p, c0, shared_tail ? 2 : 2 * ((kc_run + 1) >> 1), shared_tail ? 2 : 2 * (kc_run >> 1), v);
        }
        if constexpr (RUNS) {
          if (run) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += sums[(c0 + i) * kUmmaRows];
          }
        }
        if constexpr (KIND == I8_ROW) {
          if (p.splits == 1) {   // (with K split, the scale multiplies the sum of the partials instead)
            const float rs = row_scales[n];
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] *= rs;
          }
        }
        if (p.splits > 1) {
          // K is split over the CTAs of a cluster: the f32 partial sums go to shared memory (the rings are free: every MMA is done),
          // [token][128 features]
#pragma unroll
          for (int i = 0; i < 16; ++i) part_s[(c0 + i) * kUmmaRows + 32 * q4 + lane] = v[i];
        } else if (p.swiglu) {
          // A gate row's up row sits eight lanes on (interleaved rows), or sixteen (halves: lanes 0..15 hold a gate block, 16..31 its
          // up block).  Of every two columns the gate lanes finish the first, the up lanes the second.
          const int away = p.swiglu == 2 ? 16 : 8;
          const bool is_up = lane & away;
          const int o_col = p.swiglu == 2 ? (n >> 5) * 16 + (lane & 15) : (n >> 4) * 8 + (lane & 7);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float got = __shfl_xor_sync(0xffffffffu, is_up ? v[i] : v[i + 1], away);
            const float g = is_up ? got : v[i], up = is_up ? v[i + 1] : got;
            const int m = mt + c0 + i + is_up;
            const float act = g * (1.0f / (1.0f + expf(-g))) * up;   // the formula of swiglu_kernel, term for term
            if (m < m_end) {
              if (p.y_bf16) reinterpret_cast<__nv_bfloat16*>(p.y)[(size_t)m * p.ldy + o_col] = __float2bfloat16_rn(act);
              else reinterpret_cast<float*>(p.y)[(size_t)m * p.ldy + o_col] = act;
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int m = mt + c0 + i;
            if (m < m_end) {
              if (p.y_bf16) reinterpret_cast<__nv_bfloat16*>(p.y)[(size_t)m * p.ldy + n] = __float2bfloat16_rn(v[i]);
              else reinterpret_cast<float*>(p.y)[(size_t)m * p.ldy + n] = v[i];
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_d, 512);
  if (p.splits > 1) {
    // Every CTA of the cluster adds up its share of the tokens over all of them, in split order (reproducible), and stores it.
    cluster_sync();
    const int m_hi = min(p.ntok, p.m_total - m0), share = (m_hi + p.splits - 1) / p.splits;
    const int t_lo = (int)blockIdx.z * share, t_n = min(share, m_hi - t_lo);
    for (int idx = threadIdx.x; idx < t_n * (kUmmaRows / 4); idx += kUmmaThreads) {
      const int t = t_lo + idx / (kUmmaRows / 4), r = idx % (kUmmaRows / 4) * 4;
      if (p.swiglu && (r & 8)) continue;                       // up rows are folded into their gate rows
      float4 sum = cluster_sum(part_s + t * kUmmaRows + r, p.splits);
      const int n = blockIdx.x * kUmmaRows + r;
      int o_col = n;
      if constexpr (KIND == I8_ROW) sum = times(sum, row_scales + n);
      if (p.swiglu) {
        float4 up = cluster_sum(part_s + t * kUmmaRows + r + 8, p.splits);
        if constexpr (KIND == I8_ROW) up = times(up, row_scales + n + 8);
        sum.x = sum.x * (1.0f / (1.0f + expf(-sum.x))) * up.x;
        sum.y = sum.y * (1.0f / (1.0f + expf(-sum.y))) * up.y;
        sum.z = sum.z * (1.0f / (1.0f + expf(-sum.z))) * up.z;
        sum.w = sum.w * (1.0f / (1.0f + expf(-sum.w))) * up.w;
        o_col = (n >> 4) * 8 + (n & 7);
      }
      const size_t o = (size_t)(m0 + t) * p.ldy + o_col;
      const __nv_bfloat162 b0 = __floats2bfloat162_rn(sum.x, sum.y), b1 = __floats2bfloat162_rn(sum.z, sum.w);
      if (p.y_bf16) {
        __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(p.y) + o;
        if (p.y_vec4) {
          *reinterpret_cast<uint2*>(y) = make_uint2(*reinterpret_cast<const uint32_t*>(&b0), *reinterpret_cast<const uint32_t*>(&b1));
        } else {
          y[0] = b0.x; y[1] = b0.y; y[2] = b1.x; y[3] = b1.y;
        }
      } else {
        float* y = reinterpret_cast<float*>(p.y) + o;
        if (p.y_vec4) {
          *reinterpret_cast<float4*>(y) = sum;
        } else {
          y[0] = sum.x; y[1] = sum.y; y[2] = sum.z; y[3] = sum.w;
        }
      }
    }
    cluster_sync();                                            // nobody leaves while its partial sums are read
  }
}

// ---- host side ------------------------------------------------------------------------------------
bool umma_supported(const tq_qweight* w, size_t m) {
  return (w->kind == TQ_Q4_F16 || w->kind == TQ_Q4_F32 || w->kind == TQ_Q8_F32 || w->kind == TQ_I8_ROW) && w->rows % kUmmaRows == 0 &&
         w->cols % kTileK == 0 && m >= 1;
}

// Fewer output tiles than this leave SMs idle, and K is split.
static bool umma_few_tiles(const tq_ctx* ctx, long long ctas) { return ctas < (ctx->sm_count * 3) / 4; }
// The limit of a kernel's shared memory belongs to the kernel, not to a context: every host thread sets the same value.
constexpr int kUmmaMaxSmem = 227 * 1024;
constexpr int kUmmaTokens = 128;   // token tile: what tensor memory leaves beside the weights

// Whether two-term products of m rows run without a split of K.
bool umma_fills_gpu(const tq_ctx* ctx, const tq_qweight* w, size_t m) {
  return !umma_few_tiles(ctx, (long long)(w->rows / kUmmaRows) * (long long)((m + kUmmaTokens - 1) / kUmmaTokens));
}

// How many clusters of `size` CTAs of this kernel the GPU holds at once (a CTA has an SM to itself, whatever its shared memory).
static int umma_clusters(tq_ctx* ctx, int size) {
  int& n = ctx->umma_clusters[size];
  if (n == 0) {
    auto kern = qgemm_umma_kernel<Q4_F16, 2>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, size);
    cfg.blockDim = dim3(kUmmaThreads);
    cfg.dynamicSmemBytes = 200 * 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)size;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kUmmaMaxSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = -1;
    }
  }
  return n;
}

// y[m, rows] = x[m, cols] . W^T through the tcgen05 kernel.  x: bf16, 16-byte aligned rows.
// With `grp`: `grp->n_groups` weight matrices stacked by rows (experts); group e multiplies rows
// offsets[e] .. +counts[e] of x (device arrays) and m is the total row count of x / y.
int launch_qgemm_umma(tq_ctx* ctx, const tq_qweight* w, const void* x_bf16, size_t ldx, size_t m, void* y, int y_dtype,
                      size_t ldy, int terms, const UmmaGroups* grp, int swiglu) {
  if (w->kind == TQ_I8_ROW) terms = 1;   // exact with one term: the row scale is applied to the accumulator
  if (!encode_tiled()) return fail(ctx, TQ_EUNSUPPORTED, "cuTensorMapEncodeTiled is not available from this driver");
  TQ_REQUIRE(ctx, umma_supported(w, m), "tcgen05 GEMM: needs rows %% 128 == 0 and cols %% 128 == 0");
  TQ_REQUIRE(ctx, ((uintptr_t)x_bf16 & 15) == 0 && (ldx * 2) % 16 == 0, "tcgen05 GEMM: activation rows must be 16-byte aligned");
  // The dequantised weights are an operand in tensor memory: per chunk of 128 k and term 64 columns, four stages with one
  // term, two with two terms, i.e. 256 columns; the other 256 hold accumulators, two at least (one per issuing warp): token tiles
  // up to 128, evened out over the tiles.
  const size_t raw_tile = 8 * (size_t)qk_tile_bytes(w->kind);
  const size_t budget = kUmmaMaxSmem - kUmmaHeader - 1024;
  const int ntok_max = kUmmaTokens;
  // Many rows, one term: a CTA takes TWO token tiles (each MMA issuer multiplies every stage with its own tile's
  // activations), so the weights are converted once per 2 x <= 192 tokens; the accumulators are 2 x 192 columns, the
  // weights (two stages) 128.  Only where that still gives about a wave of CTAs (no K split in this form).
  bool dual = false;
  int dual_ntok = 0;
  size_t n_pairs = 0;
  if (terms == 1 && !grp && m > kUmmaTokens) {
    int cap = (int)(((budget - 4 * raw_tile) / kUmmaMaxXSlots) / 256) / 16 * 16;   // two activation boxes per slot
    if (cap > 192) cap = 192;
    if (cap >= 64) {
      n_pairs = (m + 2 * (size_t)cap - 1) / (2 * (size_t)cap);
      dual_ntok = (int)(((m + 2 * n_pairs - 1) / (2 * n_pairs) + 15) / 16 * 16);
      dual = !umma_few_tiles(ctx, (long long)(w->rows / kUmmaRows) * (long long)n_pairs);
    }
  }
  const size_t rows_g = grp ? w->rows / grp->n_groups : w->rows;       // output features per group
  if (grp) TQ_REQUIRE(ctx, grp->n_groups > 0 && w->rows % grp->n_groups == 0 && rows_g % kUmmaRows == 0 && grp->counts && grp->offsets,
                      "tcgen05 GEMM: every group needs a multiple of 128 output features");
  // grouped: the token tile follows the expected rows per group (tiles past a group's rows leave at once)
  const size_t m_tile_basis = grp ? (size_t)grp->expected_rows : m;
  const size_t n_tok_tiles = dual ? n_pairs : grp ? 1 : (m + ntok_max - 1) / ntok_max;   // CTAs along the tokens
  int ntok = (int)(((m_tile_basis + n_tok_tiles - 1) / n_tok_tiles + 15) / 16 * 16);
  if (ntok > ntok_max) ntok = ntok_max;
  if (ntok < 16) ntok = 16;
  if (dual) ntok = dual_ntok;
  const int ntok_stage = dual ? 2 * ntok : ntok;   // activation rows per stage
  // Few output tiles (narrow layers, small batches) leave most SMs idle: split K over gridDim.z.
  const int base_ctas = (int)(w->rows / kUmmaRows) * (int)n_tok_tiles;
  int splits = 1;
  if (!grp && swiglu != 2 && umma_few_tiles(ctx, base_ctas)) {
    splits = ctx->sm_count / base_ctas;
    if (splits > w->n_kc / 4) splits = w->n_kc / 4;      // at least eight 64-k steps per CTA
    if (splits > kUmmaMaxSplits) splits = kUmmaMaxSplits;
    while (splits > 1 && umma_clusters(ctx, splits) < base_ctas) --splits;   // (all of them at once: one wave)
    if (splits < 1) splits = 1;
  }
  const int kc_per_split = (w->n_kc + splits - 1) / splits;
  splits = (w->n_kc + kc_per_split - 1) / kc_per_split;
  int acc_stride = 32;
  while (acc_stride < ntok) acc_stride <<= 1;
  if (ntok > 128) acc_stride = 192;
  const int a_col0 = dual ? 384 : 256, stages = terms == 2 || dual ? 2 : 4;
  int n_acc = 2;                       // a power of two, as many as tensor memory holds beside the weights
  while (!dual && n_acc < 16 && 2 * n_acc * acc_stride <= a_col0) n_acc <<= 1;
  // Two accumulators for each of two token tiles, where they fit and the sums' error shows: int8 rows with f32 results.  14336 x 4096 at 144 rows:
  // error 1.05e-6 with one, 4.3e-7 with two, as with a token tile per CTA; 26 us either way.  (A kernel that can do both costs 2048 rows 2.5 %.)
  const bool two_acc = dual && ntok <= kUmmaDualAcc && w->kind == TQ_I8_ROW && y_dtype == TQ_F32;
  if (two_acc) acc_stride = 2 * kUmmaDualAcc;
  // Clusters take fewer CTAs along K than there are idle SMs (eight at most, as many as run at once), and token tiles of 128 leave fewer idle than
  // wider ones would.  f32 results of exact products keep sums as short as an even spread of K over the idle SMs gives (limited where its
  // partial sums would outweigh the weights): after a run of that many chunks the accumulators are added up in shared memory and start anew.  Not
  // bf16 results, nor weights rounded to bf16: that rounding is a thousand times the sums' error.
  // Error, us, uncut -> cut: int4 6144 x 4096 at 64 rows 6.9e-7 -> 3.9e-7, 13.1 -> 14.7; 1024 x 14336 at 48 rows 6.1e-7 -> 2.7e-7, 11.6 -> 13.9;
  // int8 5120 x 7168 at 144 rows 8.6e-7 -> 2.2e-7, 27.6 -> 32.6.  A cut costs 1 us: the products of the next run wait for it.
  int run_kc = 0;
  if (!grp && !dual && y_dtype == TQ_F32 && (terms == 2 || w->kind == TQ_I8_ROW)) {
    const size_t wide = terms == 2 ? kUmmaTokens : 192;
    const long long tiles = (long long)(w->rows / kUmmaRows) * (long long)((m + wide - 1) / wide);
    if (umma_few_tiles(ctx, tiles)) {
      long long spread = ctx->sm_count / tiles;
      const long long limit = (long long)(w->tile_bytes / (m * w->rows * 8));
      if (spread > w->n_kc / 4) spread = w->n_kc / 4;
      if (spread > 16) spread = 16;
      if (spread > limit) spread = limit;
      if (spread < 1) spread = 1;
      // (two terms and up to 32 rows: four accumulators were enough; eight are there, for twice the chunks)
      const int kc = (int)((w->n_kc + spread - 1) / spread) * (terms == 2 && n_acc == 8 ? 2 : 1);
      if (kc < kc_per_split) run_kc = kc < 2 ? 2 : kc & ~1;
    }
  }
  const size_t sum_bytes = run_kc ? (size_t)ntok * kUmmaRows * 4 : 0, ring_budget = budget - sum_bytes;
  // Shared memory: slots of activations (KX boxes of 64 k by one copy; one box with two token tiles), the rest packed tiles, whose bytes
  // in flight hide the latency of HBM: ring slots of KT = 4 k-tiles where two such fit, else 2.
  const int kx = dual ? 1 : ntok <= 64 ? 4 : 2;
  int x_slots = kx == 4 && ntok > 32 ? 3 : 4;
  if (kx == 4 && x_slots > (kc_per_split + 1) / 2) x_slots = (kc_per_split + 1) / 2;
  if (kx == 2 && (kc_per_split <= 2 || ring_budget < (size_t)x_slots * kx * umma_box_bytes(ntok_stage) + 8 * raw_tile)) x_slots = 2;   // (even: a slot is always the same issuer's)
  const size_t x_ring = (size_t)x_slots * kx * umma_box_bytes(ntok_stage);
  if (x_ring + 4 * raw_tile > ring_budget) return fail(ctx, TQ_EUNSUPPORTED, "tcgen05 GEMM: token tile of %d does not fit", ntok);
  const size_t avail = ring_budget - x_ring;
  const int kt = avail / (4 * raw_tile) >= 2 ? 4 : 2;
  int raw_stages = (int)(avail / ((size_t)kt * raw_tile));
  if (raw_stages > kUmmaMaxRawStages) raw_stages = kUmmaMaxRawStages;
  const int slots_needed = (kc_per_split + kt - 1) / kt;
  if (raw_stages > slots_needed) raw_stages = slots_needed;
  CUtensorMap map;
  if (!encode_bf16_k64_blocks(&map, x_bf16, m, w->cols, ldx, (unsigned)ntok, (unsigned)kx)) return fail(ctx, TQ_ECUDA, "cuTensorMapEncodeTiled failed");
  CUtensorMap w_map;   // the packed tiles as 128-byte lines, boxes of kt tiles of four row blocks
  if (!encode_lines128(&w_map, w->tiles, (size_t)w->n_kc * (qk_tile_bytes(w->kind) / 128), (size_t)w->n_rb, (unsigned)(kt * (qk_tile_bytes(w->kind) / 128)), 4))
    return fail(ctx, TQ_ECUDA, "cuTensorMapEncodeTiled failed");
  UmmaParams p;
  p.row_scales = w->row_scales;
  p.y = y;
  p.ldy = (long long)ldy;
  p.m_total = (int)m;
  p.n_rows = (int)rows_g;
  p.g_counts = grp ? grp->counts : nullptr;
  p.g_offsets = grp ? grp->offsets : nullptr;
  p.n_groups = grp ? grp->n_groups : 1;
  p.kc_total = w->n_kc;
  p.ntok = ntok;
  p.acc_stride = acc_stride;
  p.n_acc = n_acc;
  p.a_col0 = a_col0;
  p.y_bf16 = y_dtype == TQ_BF16;
  TQ_REQUIRE(ctx, swiglu != 2 || w->kind != TQ_I8_ROW, "tcgen05 GEMM: gate and up halves with row scales");
  p.swiglu = swiglu;
  p.err = ctx->dev_err;
  p.splits = splits;
  p.kc_per_split = kc_per_split;
  p.run_kc = run_kc;
  p.y_vec4 = ldy % 4 == 0 && ((uintptr_t)y & (p.y_bf16 ? 7 : 15)) == 0;
  p.stages = stages;
  p.x_slots = x_slots;
  p.kx = kx;
  p.raw_stages = raw_stages;
  p.kt = kt;
  const size_t smem = umma_smem_bytes(w->kind, x_ring, raw_stages * kt) + sum_bytes;
  if (smem > kUmmaMaxSmem) return fail(ctx, TQ_EUNSUPPORTED, "tcgen05 GEMM: %zu bytes of shared memory needed", smem);
  dim3 grid((unsigned)(rows_g / kUmmaRows), (unsigned)((m + ntok_stage - 1) / ntok_stage), (unsigned)splits);
  if (grp) {
    grid.y = (unsigned)(m / ntok + (size_t)(grp->max_active < grp->n_groups ? grp->max_active : grp->n_groups));   // (a last tile per group with rows)
    grid.z = 1;
  }
  auto go = [&](auto kern) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kUmmaMaxSmem);
    if (e != cudaSuccess) return e;
    if (splits > 1) return launch_k_cluster(ctx, kern, grid, dim3(kUmmaThreads), smem, dim3(1, 1, splits), map, w_map, p);
    return launch_k(ctx, kern, grid, dim3(kUmmaThreads), smem, map, w_map, p);
  };
  cudaError_t e;
  if (dual) {
    if (splits != 1) return fail(ctx, TQ_EUNSUPPORTED, "tcgen05 GEMM: two token tiles per CTA with K split");
    if (w->kind == TQ_I8_ROW) e = two_acc ? go(qgemm_umma_kernel<I8_ROW, 1, 2>) : go(qgemm_umma_kernel<I8_ROW, 1, 1>);
    else if (w->kind == TQ_Q4_F16) e = go(qgemm_umma_kernel<Q4_F16, 1, 1>);
    else if (w->kind == TQ_Q8_F32) e = go(qgemm_umma_kernel<Q8_F32, 1, 1>);
    else e = go(qgemm_umma_kernel<Q4_F32, 1, 1>);
  } else if (run_kc) {
    if (w->kind == TQ_I8_ROW) e = go(qgemm_umma_kernel<I8_ROW, 1, 0, true>);
    else if (w->kind == TQ_Q4_F16) e = go(qgemm_umma_kernel<Q4_F16, 2, 0, true>);
    else if (w->kind == TQ_Q8_F32) e = go(qgemm_umma_kernel<Q8_F32, 2, 0, true>);
    else e = go(qgemm_umma_kernel<Q4_F32, 2, 0, true>);
  } else if (w->kind == TQ_I8_ROW) e = go(qgemm_umma_kernel<I8_ROW, 1>);
  else if (w->kind == TQ_Q4_F16) e = terms == 2 ? go(qgemm_umma_kernel<Q4_F16, 2>) : go(qgemm_umma_kernel<Q4_F16, 1>);
  else if (w->kind == TQ_Q8_F32) e = terms == 2 ? go(qgemm_umma_kernel<Q8_F32, 2>) : go(qgemm_umma_kernel<Q8_F32, 1>);
  else e = terms == 2 ? go(qgemm_umma_kernel<Q4_F32, 2>) : go(qgemm_umma_kernel<Q4_F32, 1>);
  TQ_CUDA(ctx, e);
  return TQ_OK;
}

// Grouped entry for the other translation units: experts stacked by rows, rows of x / y grouped by expert.
int launch_qgemm_umma_grouped(tq_ctx* ctx, const tq_qweight* w, int n_groups, const void* x_bf16, size_t ldx, size_t m_total,
                              const int* counts, const int* offsets, int max_active, int expected_rows,
                              void* y, int y_dtype, size_t ldy, int terms, int swiglu) {
  UmmaGroups g;
  g.n_groups = n_groups;
  g.counts = counts;
  g.offsets = offsets;
  g.max_active = max_active;
  g.expected_rows = expected_rows;
  return launch_qgemm_umma(ctx, w, x_bf16, ldx, m_total, y, y_dtype, ldy, terms, &g, swiglu);
}

bool umma_grouped_supported(const tq_qweight* w, int n_groups) {
  return (w->kind == TQ_Q4_F16 || w->kind == TQ_Q4_F32) && n_groups > 0 && w->rows % n_groups == 0 &&
         (w->rows / n_groups) % kUmmaRows == 0 && w->cols % kTileK == 0;
}

}  // namespace tq
