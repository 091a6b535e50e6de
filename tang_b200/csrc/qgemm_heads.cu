// Many small weights of one shape stacked by rows, each with its own few activation rows and a short K: the per-head products
// around the latent attention (128 x [512, 128] and 128 x [128, 512] int8 matrices, 1 to 64 rows).
//
//     y[m, e, n] = sum_k x[m, e, k] * q[e, n, k] * scale[e, n, k / 32]      (crates/tang-infer/src/quantize.rs:227-289, per head)
//
// A warp owns one 16-row block of one weight, up to sixteen activation rows and all of K: it reads the fragment tiles straight into
// registers, the activation fragments straight from global memory (a head's rows are a few KB that its warps share in L1), and stores
// its results.  No shared memory, no barrier, nothing to park.  Bound: the latency of two dependent loads, behind which the bytes
// (8.4 MB) hide.  More rows are more CTAs that read the tiles from L2: all of 64 rows in one warp took 18.6 and 17.8 us (registers).
// The general kernel spends its time on setting up a ring per CTA for one or four tiles of K.  int8, [512, 128] and [128, 512], us, the
// general kernel -> this one: 128 heads, one row 8.1 / 6.6 -> 4.8 / 3.1, sixteen 16.9 / 15.3 -> 6.4 / 7.4, 64 54.7 / 46.6 -> 15.7 / 15.4;
// 16 heads, one row, [512, 128] 4.6 -> 3.3.  Errors of f32 results of K = 512 against 64 bits 5.3e-8 -> 5.0e-8.
#include "internal.h"
#include "qtile.cuh"

namespace tq {

struct QHeadsParams {
  const uint8_t* tiles;       // [groups][rb_g][n_kc][tile bytes]
  const float* row_scales;    // I8_ROW only: [groups][16 rb_g]
  const __nv_bfloat16* x;
  void* y;
  long long ldx, ldy, x_stride, y_stride;   // elements between rows, and between groups
  int n_blocks, rb_g, n_kc, mx, y_bf16;     // n_blocks: row blocks of all groups
};

constexpr int kHeadsWarps = 8;

// ONE: K is one chunk
template <int KIND, int NT, bool ONE>
__global__ void __launch_bounds__(32 * kHeadsWarps) qgemm_heads_kernel(const QHeadsParams p) {
  constexpr bool kIs8 = KIND == Q8_F32 || KIND == I8_ROW;
  constexpr int WB = kIs8 ? 2048 : 1024, TB = WB + (KIND == Q4_F16 ? 128 : KIND == I8_ROW ? 0 : 256), NV = WB / 512;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int blk = blockIdx.x * kHeadsWarps + (threadIdx.x >> 5);
  const bool live = blk < p.n_blocks;
  const int e = live ? blk / p.rb_g : 0, rb = live ? blk - e * p.rb_g : 0;
  const uint8_t* tile = p.tiles + (size_t)(live ? blk : 0) * p.n_kc * TB;
  uint4 w[NV];
  auto load = [&](const uint8_t* src) {
#pragma unroll
    for (int i = 0; i < NV; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(src + 512 * i) + lane);
  };
  load(tile);                       // the weights do not depend on the previous kernel of the stream
  pdl_wait();
  pdl_launch_dependents();
  if (!live) return;
  const int m0 = 16 * blockIdx.y;
  const __nv_bfloat16* x = p.x + (size_t)e * p.x_stride + 8 * t;
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 1
  for (int kc = 0; kc < (ONE ? 1 : p.n_kc); ++kc, tile += TB) {
    float sc[2][4];
    if constexpr (KIND == Q4_F16) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(tile + WB + h * 64 + g * 8));
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
        sc[h][0] = a.x; sc[h][1] = a.y; sc[h][2] = b.x; sc[h][3] = b.y;
      }
    } else if constexpr (KIND != I8_ROW) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(tile + WB + h * 128 + g * 16));
        sc[h][0] = v.x; sc[h][1] = v.y; sc[h][2] = v.z; sc[h][3] = v.w;
      }
    }
    tile_sums<KIND, NT, ONE>(
        acc, sc,
        [&](int j, uint32_t (&a)[2][4]) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if constexpr (kIs8) {
              const uint4& v = w[2 * h + (j >> 1)];
              dequant_i8_words(j & 1 ? v.z : v.x, j & 1 ? v.w : v.y, a[h]);
            } else {
              const uint4& v = w[h];
              dequant_q4_word(j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w, a[h]);
            }
          }
        },
        [&](int i, int j) {
          return m0 + 8 * i + g < p.mx ? *reinterpret_cast<const uint4*>(x + (size_t)(m0 + 8 * i + g) * p.ldx + kc * kTileK + 32 * j) : make_uint4(0u, 0u, 0u, 0u);
        });
    if (!ONE && kc + 1 < p.n_kc) load(tile + TB);
  }
  const int n0 = 16 * rb + g;
  float s[2] = {1.f, 1.f};
  if constexpr (KIND == I8_ROW) {
    s[0] = p.row_scales[(size_t)e * 16 * p.rb_g + n0];
    s[1] = p.row_scales[(size_t)e * 16 * p.rb_g + n0 + 8];
  }
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int m = m0 + 8 * i + 2 * t + (c & 1);
      if (m >= p.mx) continue;
      const size_t o = (size_t)m * p.ldy + (size_t)e * p.y_stride + n0 + 8 * (c >> 1);
      const float v = acc[i][c] * s[c >> 1];
      if (p.y_bf16) static_cast<__nv_bfloat16*>(p.y)[o] = __float2bfloat16_rn(v);
      else static_cast<float*>(p.y)[o] = v;
    }
}

template <int KIND, bool ONE>
static cudaError_t heads_launch(tq_ctx* ctx, const QHeadsParams& p) {
  const dim3 grid((unsigned)((p.n_blocks + kHeadsWarps - 1) / kHeadsWarps), (unsigned)((p.mx + 15) / 16)), block(32 * kHeadsWarps);
  if (p.mx <= 8) return launch_k(ctx, qgemm_heads_kernel<KIND, 1, ONE>, grid, block, 0, p);
  return launch_k(ctx, qgemm_heads_kernel<KIND, 2, ONE>, grid, block, 0, p);
}
template <int KIND>
static cudaError_t heads_launch(tq_ctx* ctx, const QHeadsParams& p) {
  return p.n_kc == 1 ? heads_launch<KIND, true>(ctx, p) : heads_launch<KIND, false>(ctx, p);
}

// `n_groups` weights stacked by rows (a multiple of 16 each), group e's rows start x_stride / y_stride elements into x / y; x 16-byte
// aligned in base, row and group strides, K a multiple of 128 (the caller's checks).  false: the shape is for another kernel.
bool launch_qgemm_heads(tq_ctx* ctx, const tq_qweight* w, int n_groups, const void* x_bf16, size_t ldx, int mx, long long x_stride, long long y_stride,
                        void* y, int y_dtype, size_t ldy, int* status) {
  // A warp walks K alone, so enough row blocks to fill the GPU with warps: [128, 512] at sixteen rows, 256 row blocks 7.3 us against 4.3
  // with the general kernel, 512 7.4 against 7.8 (at one to eight rows both sides are within 1 us from 128 row blocks on).  Up to four
  // chunks is what the layer's widths (128 and 512) need; longer K would be faster here as well (64 heads, sixteen rows, [512, 640]
  // 11.4 us against 35.1, [512, 1024] 16.5 against 24.4), but no configuration has it.
  if (mx < 1 || mx > 64 || w->n_kc > 4 || w->n_rb < 2 * ctx->sm_count) return false;
  QHeadsParams p;
  p.tiles = w->tiles;
  p.row_scales = w->row_scales;
  p.x = static_cast<const __nv_bfloat16*>(x_bf16);
  p.y = y;
  p.ldx = (long long)ldx;
  p.ldy = (long long)ldy;
  p.x_stride = x_stride;
  p.y_stride = y_stride;
  p.n_blocks = w->n_rb;
  p.rb_g = w->n_rb / n_groups;
  p.n_kc = w->n_kc;
  p.mx = mx;
  p.y_bf16 = y_dtype == TQ_BF16;
  cudaError_t e;
  switch (w->kind) {
    case TQ_Q4_F32: e = heads_launch<Q4_F32>(ctx, p); break;
    case TQ_Q4_F16: e = heads_launch<Q4_F16>(ctx, p); break;
    case TQ_Q8_F32: e = heads_launch<Q8_F32>(ctx, p); break;
    default: e = heads_launch<I8_ROW>(ctx, p); break;
  }
  *status = e == cudaSuccess ? TQ_OK : fail(ctx, TQ_ECUDA, "per-head product launch failed: %s", cudaGetErrorString(e));
  return true;
}

}  // namespace tq
