// Quantised linear layer for 9 to 16 activation rows: weights from HBM through a private ring of every warp, straight into
// mma.sync fragments.
//
//     y[m, n] = sum_k x[m, k] * q[n, k] * scale[n, k / 32]        (crates/tang-infer/src/quantize.rs:227-289)
//
// Bound: instructions and their latencies rather than bytes (14336 x 4096 at 12 rows under ncu: issue slots 48 % busy, ALU 34 %,
// tensor pipe 20 %, DRAM 18 %).  So what stands around the products is kept short:
//   * K is cut into slabs of `skc` 128-k chunks (one slab where the activations fit); a CTA belongs to one slab and keeps its
//     slab of the activation rows in shared memory for its whole life: one read of x per CTA, no activation pipeline;
//   * the slab's tiles, numbered (row block, chunk), are cut evenly over all WARPS of its CTAs.  A warp walks its contiguous
//     range alone: it copies its own tiles into its own ring (cp.async, D stages), so there is no barrier between warps and no
//     producer, and every warp has D - 1 tiles in flight;
//   * a fragment tile is read from the ring as the A operand (qlayout.cuh), unpacked to exact bf16 integers, multiplied
//     with mma.sync, and the 32-block's scale multiplies the f32 partial sum: products are exact, only f32 sums round (qtile.cuh);
//   * a (row block, slab) piece that does not hold all of K is parked as f32 fragments; the warp whose tiles complete a row
//     block (a counter of tiles) adds the parked pieces in slab order, then in warp order: the same bits whoever that is.
//     Nobody waits for anybody.  (Pieces of one CTA meeting in shared memory behind a CTA barrier at the end measured slower:
//     18.5 against 16.0 us at 14336 x 4096, 24.1 against 18.9 at 4096 x 14336, where it now takes 16.6 and 17.2.)
// Measured, 12 rows, f32 results, against the general kernel: 14336 x 4096 Q4 22.1 -> 16.6 us, 4096 x 14336 27.7 -> 17.2,
// 6144 x 4096 17.0 -> 11.0, int8 24576 x 1536 32.3 -> 15.4, int8 7168 x 16384 67.9 -> 34.2.  Errors against 64 bits, relative to the
// result's norm, Q4: 1.11e-7 -> 7.6e-8, 1.46e-7 -> 7.9e-8, 9.3e-8 -> 6.5e-8; int8 6.3e-8 -> 6.2e-8, 14336 x 4096 8.3e-8 -> 6.9e-8.
#pragma once

#include <cfloat>

#include "common.cuh"
#include "qlayout.cuh"
#include "qtile.cuh"

namespace tq {

struct QWrParams {
  const uint8_t* tiles;       // fragment tiles, [n_rb][kc_total][tile bytes]
  const float* row_scales;    // I8_ROW only
  const __nv_bfloat16* x;     // [mx][ldx], rows 16-byte aligned, kc_total * 128 valid elements per row
  const float* residual;      // optional f32 [mx][ldy] added before the store (may be y)
  void* y;                    // [mx][ldy] f32 or bf16
  long long ldx, ldy;
  int n_rows, n_rb, kc_total, mx;
  int y_bf16, swiglu;         // swiglu: gate/up rows interleaved by eight; silu(gate) * up, n_rows / 2 values per row
  int skc, n_slabs, cps;      // chunks per slab, slabs, CTAs per slab
  float* part;                // parked pieces: [n_slabs][n_rb] that start a slab, then one per warp, [n_slabs][cps * 16]
  int* counters;              // [n_rb] tiles summed so far, zero between launches
};

constexpr int kWrRows = 16, kWrNT = kWrRows / 8, kWrWarps = 16;
constexpr int kWrPiece = kWrNT * 128;                                     // floats
__host__ __device__ inline int qwr_x_stride(int skc) { return skc * kTileK * 2 + 64; }   // 64 (mod 128) bytes: no bank conflicts

template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16_hint(uint32_t dst, const void* src, uint64_t pol) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(pol) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
// Stores a finished row block: acc[i][c] holds row g (c < 2) or g + 8 of it, activation rows 8 i + 2 t + c % 2.
template <int KIND>
__device__ __forceinline__ void wr_store(const QWrParams& p, float (&acc)[kWrNT][4], int rb, int g, int t) {
  const int n0 = rb * kTileRows + g;
  float s0 = 1.f, s1 = 1.f;
  if constexpr (KIND == I8_ROW) {
    s0 = n0 < p.n_rows ? p.row_scales[n0] : 0.f;
    s1 = n0 + 8 < p.n_rows ? p.row_scales[n0 + 8] : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kWrNT; ++i)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int m = 8 * i + 2 * t + c;
      if (m >= p.mx) continue;
      float v0 = acc[i][c], v1 = acc[i][2 + c];
      if constexpr (KIND == I8_ROW) {
        v0 *= s0;
        v1 *= s1;
      }
      if (p.swiglu) {
        if (n0 + 8 < p.n_rows) {
          const float v = v0 * (1.0f / (1.0f + expf(-v0))) * v1;
          const size_t o = (size_t)m * p.ldy + rb * 8 + g;
          if (p.y_bf16) static_cast<__nv_bfloat16*>(p.y)[o] = __float2bfloat16_rn(v);
          else static_cast<float*>(p.y)[o] = v;
        }
        continue;
      }
      const size_t o = (size_t)m * p.ldy + n0;
      if (n0 < p.n_rows) {
        if (p.residual) v0 += p.residual[o];
        if (p.y_bf16) static_cast<__nv_bfloat16*>(p.y)[o] = __float2bfloat16_rn(v0);
        else static_cast<float*>(p.y)[o] = v0;
      }
      if (n0 + 8 < p.n_rows) {
        if (p.residual) v1 += p.residual[o + 8];
        if (p.y_bf16) static_cast<__nv_bfloat16*>(p.y)[o + 8] = __float2bfloat16_rn(v1);
        else static_cast<float*>(p.y)[o + 8] = v1;
      }
    }
}

template <int KIND, int D>
__global__ void __launch_bounds__(32 * kWrWarps, 1) qgemm_wr_kernel(const QWrParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr bool kIs8 = KIND == Q8_F32 || KIND == I8_ROW;
  constexpr int WB = kIs8 ? 2048 : 1024;                                     // weight bytes of a tile; scales follow
  constexpr int SB = KIND == Q4_F16 ? 128 : KIND == I8_ROW ? 0 : 256;
  constexpr int TB = WB + SB, W = kWrWarps, NT = kWrNT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int slab = blockIdx.x % p.n_slabs, cta = blockIdx.x / p.n_slabs;
  const int kc0 = slab * p.skc, skc = min(p.skc, p.kc_total - kc0);
  const long long total = (long long)p.n_rb * skc;
  const int n_w = p.cps * W, w_id = cta * W + warp;
  const int lo = (int)(total * w_id / n_w), hi = (int)(total * (w_id + 1) / n_w);            // this warp's tiles
  const int xs_stride = qwr_x_stride(p.skc);
  const uint32_t x_s = smem_u32(smem);
  const uint32_t ring = x_s + (uint32_t)(kWrRows * xs_stride) + (uint32_t)(warp * (D * TB));
  const uint64_t pol = l2_policy_evict_first();

  // ---- copies of this warp's tiles: (fb, fc) is the next tile to ask for
  int fb = lo / skc, fc = lo - fb * skc, fslot = 0, left = hi - lo;
  auto fetch = [&]() {
    if (left > 0) {
      --left;
      const uint32_t dst = ring + (uint32_t)(fslot * TB) + 16u * lane;
      const uint8_t* src = p.tiles + ((size_t)fb * p.kc_total + kc0 + fc) * TB + 16 * lane;
#pragma unroll
      for (int i = 0; i < WB / 512; ++i) cp_async16_hint(dst + 512 * i, src + 512 * i, pol);
      if (SB > 0 && lane < SB / 16) cp_async16_hint(dst + WB, src + WB, pol);
      if (++fc == skc) {
        fc = 0;
        ++fb;
      }
      if (++fslot == D) fslot = 0;
    }
    cp_async_commit();
  };
  // the weights do not depend on the previous kernel of the stream; the activations do
#pragma unroll
  for (int i = 0; i < D - 1; ++i) fetch();
  pdl_wait();
  pdl_launch_dependents();
  {
    const int per_row = skc * (kTileK / 8);
    for (int i = threadIdx.x; i < p.mx * per_row; i += 32 * W) {
      const int m = i / per_row, c = i - m * per_row;
      cp_async16(x_s + (uint32_t)(m * xs_stride + 16 * c), p.x + (size_t)m * p.ldx + (size_t)kc0 * kTileK + 8 * c);
    }
    // rows that only fill the last column tile read as zeros
    const int pad16 = xs_stride / 16;
    for (int i = threadIdx.x; i < (kWrRows - p.mx) * pad16; i += 32 * W)
      *reinterpret_cast<uint4*>(smem + (size_t)p.mx * xs_stride + 16 * (size_t)i) = make_uint4(0u, 0u, 0u, 0u);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  }

  float acc[NT][4];
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  };
  clear();
  const uint32_t x_lane = x_s + (uint32_t)(g * xs_stride + 16 * t);
  int rb = lo / skc, kc = lo - rb * skc, slot = 0, done = 0;
#pragma unroll 1
  for (int u = lo; u < hi; ++u) {
    cp_async_wait<D - 2>();
    __syncwarp();                       // every lane's copies of this tile have landed, and every lane is done with the tile before
    fetch();
    // ---- one tile of 16 rows x 128 k
    const uint32_t tile = ring + (uint32_t)(slot * TB);
    const uint32_t xk = x_lane + (uint32_t)(kc * (2 * kTileK));
    float sc[2][4];                     // scales of rows g, g + 8 for the four 32-blocks
    uint4 w4[2];
    if constexpr (KIND == Q4_F16) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint2 v = lds64(tile + WB + h * 64 + g * 8);
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
        sc[h][0] = a.x; sc[h][1] = a.y; sc[h][2] = b.x; sc[h][3] = b.y;
      }
    } else if constexpr (KIND != I8_ROW) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 v = lds128(tile + WB + h * 128 + g * 16);
        sc[h][0] = __uint_as_float(v.x); sc[h][1] = __uint_as_float(v.y);
        sc[h][2] = __uint_as_float(v.z); sc[h][3] = __uint_as_float(v.w);
      }
    }
    if constexpr (!kIs8) {
      w4[0] = lds128(tile + 16 * lane);
      w4[1] = lds128(tile + 512 + 16 * lane);
    }
    tile_sums<KIND, NT>(
        acc, sc,
        [&](int j, uint32_t (&a)[2][4]) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if constexpr (kIs8) {
              const uint2 v = lds64(tile + h * 1024 + (j >> 1) * 512 + 16 * lane + 8 * (j & 1));
              dequant_i8_words(v.x, v.y, a[h]);
            } else {
              dequant_q4_word(j == 0 ? w4[h].x : j == 1 ? w4[h].y : j == 2 ? w4[h].z : w4[h].w, a[h]);
            }
          }
        },
        [&](int i, int j) { return lds128(xk + (uint32_t)(8 * i * xs_stride + 64 * j)); });
    if (++slot == D) slot = 0;
    ++done;
    if (++kc < skc && u + 1 < hi) continue;
    // ---- this warp's piece of the row block is finished: `done` tiles of slab `slab`
    bool mine = done == p.kc_total;     // ... which are all there are
    if (!mine) {
      const size_t heads = (size_t)p.n_slabs * p.n_rb;
      const bool first = done == kc;                   // the piece starts at the slab's first chunk
      float* dst = p.part + (first ? (size_t)slab * p.n_rb + rb : heads + (size_t)slab * n_w + w_id) * kWrPiece + 4 * lane;
#pragma unroll
      for (int i = 0; i < NT; ++i) __stcg(reinterpret_cast<float4*>(dst + i * 128), make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
      __threadfence();
      __syncwarp();
      int seen = 0;
      if (lane == 0) seen = atomicAdd(p.counters + rb, done);
      seen = __shfl_sync(0xffffffffu, seen, 0);
      mine = seen + done == p.kc_total;
      if (mine) {
        __threadfence();
        if (lane == 0) p.counters[rb] = 0;
        clear();
        // What each addition rounds away is kept aside and added last (two-sum, Knuth): the pieces of a sum without cancellation
        // are as large as the result, and up to a dozen of them one after the other would cost more than all additions before.
        float lost[NT][4] = {};
        auto add = [&](float& a, float& low, float v) {
          const float sum = a + v, b = sum - a;
          low += (a - (sum - b)) + (v - b);
          a = sum;
        };
        int first_w = 0, last_w = 0;          // of slab `lane` of these 32: owners of the first and the last tile of the row block
        int s = 0, w0 = 0, w1 = 0, wi = 0;    // the next piece: slab s, warp wi of w0 .. w1
        auto enter = [&]() {
          if ((s & 31) == 0) {
            const int ks = min(p.skc, p.kc_total - min(s + lane, p.n_slabs - 1) * p.skc);
            const long long tot = (long long)p.n_rb * ks, f0 = (long long)rb * ks;
            first_w = (int)(((f0 + 1) * n_w - 1) / tot);
            last_w = (int)(((f0 + ks) * n_w - 1) / tot);
          }
          wi = w0 = __shfl_sync(0xffffffffu, first_w, s & 31);
          w1 = __shfl_sync(0xffffffffu, last_w, s & 31);
        };
        enter();
        while (s < p.n_slabs) {
          float4 v[4][NT];                    // four pieces in flight
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const bool any = s < p.n_slabs;
            const float* src = p.part + (wi == w0 ? (size_t)s * p.n_rb + rb : heads + (size_t)s * n_w + wi) * kWrPiece + 4 * lane;
#pragma unroll
            for (int i = 0; i < NT; ++i) v[k][i] = any ? __ldcg(reinterpret_cast<const float4*>(src + i * 128)) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (any && ++wi > w1 && ++s < p.n_slabs) enter();
          }
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < NT; ++i) {
              add(acc[i][0], lost[i][0], v[k][i].x);
              add(acc[i][1], lost[i][1], v[k][i].y);
              add(acc[i][2], lost[i][2], v[k][i].z);
              add(acc[i][3], lost[i][3], v[k][i].w);
            }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (fabsf(acc[i][c]) <= FLT_MAX) acc[i][c] += lost[i][c];      // (behind an infinity `lost` is NaN)
      }
    }
    if (mine) wr_store<KIND>(p, acc, rb, g, t);
    clear();
    done = 0;
    if (kc >= skc) {
      kc = 0;
      ++rb;
    }
  }
}

}  // namespace tq
