// Launcher of the quantised linear layer for 9 to 16 rows (qgemm_wr.cuh).
#include "internal.h"
#include "qgemm_wr.cuh"

namespace tq {

constexpr int wr_depth(int kind) { return kind == Q8_F32 || kind == I8_ROW ? 4 : 8; }   // ring stages of a warp: about 9 KB

template <int KIND>
static cudaError_t wr_launch(tq_ctx* ctx, const QWrParams& p, unsigned grid, size_t smem) {
  auto kern = qgemm_wr_kernel<KIND, wr_depth(KIND)>;
  static bool done[64] = {};   // per device; the same value from every thread
  if (!done[ctx->device & 63]) {
    if (cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)) return e;
    done[ctx->device & 63] = true;
  }
  return launch_k(ctx, kern, dim3(grid), dim3(32 * kWrWarps), smem, p);
}

// Launches the kernel when it takes the shape (then *status is the result); false: the caller uses another one.
bool launch_qgemm_wr(tq_ctx* ctx, const tq_qweight* w, const void* x_bf16, size_t ldx, size_t m, void* y, int y_dtype, size_t ldy,
                     const float* residual, bool swiglu, int* status) {
  // Below nine rows the persistent kernels (one column tile of mma.sync) are faster, above sixteen the tcgen05 kernel: 24.4 us
  // against 23.2 here at 24 rows and 28.0 at 32 (14336 x 4096).
  if (m < 9 || m > (size_t)kWrRows || w->cols != (size_t)w->n_kc * kTileK || ldx % 8 != 0 || ((uintptr_t)x_bf16 & 15) != 0 || w->n_rb > kWrCounters)
    return false;
  // Little to stream: the general kernel, which parks nothing and counts nothing (12 rows: 2048 x 2048 Q4 4.0 us against 7.4, 1536 x 7168
  // int8 8.7 against 13.2; at 42 tiles per SM, 3072 x 4096, 10.9 against 10.1 and 11.7 against 10.7, but at 9 rows 6.3 against 9.9).
  // Its launcher has a rule for larger ones too (qlinear.cu).
  if ((long long)w->n_rb * w->n_kc < 50LL * ctx->sm_count) return false;
  QWrParams p;
  // The widest slabs that fit: every slab boundary is one more piece to park per row block (12 rows, Q4 14336 x 4096: 16.6 us with
  // the two slabs that fit, 20.3 with four, 27.4 with eight; int8 7168 x 16384: 34.2 with six, 41.2 with twelve, 67.7 with 24).
  const size_t ring = (size_t)kWrWarps * wr_depth(w->kind) * qk_tile_bytes(w->kind);
  const int skc_max = (int)(((227 * 1024 - ring) / kWrRows - 64) / (2 * kTileK));
  p.n_slabs = (w->n_kc + skc_max - 1) / skc_max;
  p.skc = (w->n_kc + p.n_slabs - 1) / p.n_slabs;
  p.n_slabs = (w->n_kc + p.skc - 1) / p.skc;
  p.cps = ctx->sm_count / p.n_slabs;
  const long long least = (long long)w->n_rb * (w->n_kc - (p.n_slabs - 1) * p.skc);   // tiles of the shortest slab
  if (p.cps > least / (2 * kWrWarps)) p.cps = (int)(least / (2 * kWrWarps));
  if (p.cps < 1) return false;       // (so every warp has a tile: the bookkeeping of the pieces relies on it)
  const size_t smem = ring + (size_t)kWrRows * qwr_x_stride(p.skc);
  if ((size_t)p.n_slabs * (w->n_rb + p.cps * kWrWarps) * kWrPiece * sizeof(float) > kWrPartBytes) return false;
  p.tiles = w->tiles;
  p.row_scales = w->row_scales;
  p.x = static_cast<const __nv_bfloat16*>(x_bf16);
  p.residual = residual;
  p.y = y;
  p.ldx = (long long)ldx;
  p.ldy = (long long)ldy;
  p.n_rows = (int)w->rows;
  p.n_rb = w->n_rb;
  p.kc_total = w->n_kc;
  p.mx = (int)m;
  p.y_bf16 = y_dtype == TQ_BF16;
  p.swiglu = swiglu ? 1 : 0;
  p.part = ctx->wr_part;
  p.counters = ctx->wr_counters;
  const unsigned grid = (unsigned)(p.n_slabs * p.cps);
  cudaError_t e;
  switch (w->kind) {
    case TQ_Q4_F32: e = wr_launch<Q4_F32>(ctx, p, grid, smem); break;
    case TQ_Q4_F16: e = wr_launch<Q4_F16>(ctx, p, grid, smem); break;
    case TQ_Q8_F32: e = wr_launch<Q8_F32>(ctx, p, grid, smem); break;
    default: e = wr_launch<I8_ROW>(ctx, p, grid, smem); break;
  }
  *status = e == cudaSuccess ? TQ_OK : fail(ctx, TQ_ECUDA, "quantised linear launch failed: %s", cudaGetErrorString(e));
  return true;
}

}  // namespace tq
