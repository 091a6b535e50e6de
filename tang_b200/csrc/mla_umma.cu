// Latent-attention decode core on the 5th-generation tensor cores, for 64 heads and more per rank:
//     s_j = (q . [c_j | r_j]) * scale,   o = sum_j softmax(s)_j c_j          rows of 512 + 64 bf16, shared by all heads
//
// The 128 heads of a CTA are the UMMA M dimension.  Their f32 outputs (128 x 512) would fill all of tensor memory, so a CTA owns
// one half of the latent columns (256) and forms the scores for itself; the two CTAs of a pair are neighbours in the grid and
// read the same cache rows, the second time from L2.  Per tile of 32 positions:
//   warp 0      TMA: nine groups of 32 rows x 64 columns (128-byte swizzle) in one copy into one of three stages; the queries once (the first 256
//               columns go to tensor memory, which leaves room for the third stage: with two the copies' latency was the bound).
//               The rows of a last tile that is not full come by cp.async, zeros behind them: nothing behind a sequence's end is read;
//   warp 1      issues S = Q K^T (36 MMAs of 128 x 32 x 16), then, a tile behind, O += P V (V are the same boxes, read
//               N-major): the probabilities come from tensor memory as two bf16 terms (hi + lo, 16 significant bits, as in
//               the mma.sync kernel), one MMA of 128 x 256 x 16 each;
//   warps 4..7  a thread owns one head: it reads the head's 32 scores, takes the maximum, forms P and the row sum without any
//               exchange.  O is rescaled only when a maximum has grown by more than 2^8 (the reference of the exponentials is
//               any number near the maximum; a step published with FlashAttention-4), which is rare after the first tiles;
// Measured, 128 heads: 16 sequences of 8.7k to 16.4k positions, the attention and its merge 454 us with the mma.sync kernel -> 171 us
// (tiles of 32 positions, 1.3 us each; with two stages instead of three the attention took 296 us where it took 177).
// What bounds it now is the chain copy -> scores -> softmax -> products of a tile with three tiles in flight (shared memory is full), not
// a unit: tensor pipe 41 % of active cycles, issue slots 34 %, DRAM 15 % (16 sequences of 8192, ncu).
// Splits over the positions are merged by mla_combine_kernel.  Every wait is bounded.
#include <cfloat>

#include "internal.h"
#include "qgemm_umma.cuh"
#include "tensormap.h"

namespace tq {

constexpr int kMuTile = 32, kMuLat = 512, kMuRow = 576, kMuBoxes = kMuRow / 64, kMuHalf = kMuLat / 2;
constexpr int kMuThreads = 256, kMuFirstSoft = 4;
constexpr int kMuQBox = 128 * 128, kMuKBox = kMuTile * 128;
constexpr int kMuStage = kMuBoxes * kMuKBox;
constexpr int kMuStages = 3, kMuQTmem = 4;                           // 64-column groups of the queries that live in tensor memory
constexpr size_t kMuSmem = 2048 + (size_t)(kMuBoxes - kMuQTmem) * kMuQBox + kMuStages * (size_t)kMuStage;
// tensor-memory columns: O, two S, two (P hi, P lo), the first groups of Q
constexpr int kMuColS = kMuHalf, kMuColP = kMuColS + 2 * kMuTile, kMuColQ = kMuColP + 2 * kMuTile;
static_assert(kMuColQ + kMuQTmem * 32 <= 512, "tensor memory");
constexpr float kMuGrow = 8.f;                                       // log2 of how far a maximum may run ahead of its reference

struct MlaUmmaParams {
  const __nv_bfloat16* q;         // [B][H][576]
  const __nv_bfloat16* cache;     // sequence b from b * seq_stride on
  size_t seq_stride;
  const int* lens;
  int n_heads, n_splits, chunk;   // chunk: positions per split, a multiple of the tile
  float scale;                    // softmax scale times log2(e)
  __nv_bfloat16* out;             // [B][H][512] (n_splits == 1)
  float* part_o;                  // [B][H][n_splits][512]
  float* part_ml;                 // [B][H][n_splits][2]: reference of the exponentials in powers of two, sum
  int* err;
};

__device__ __forceinline__ void mu_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mu_ld32(uint32_t taddr, float (&v)[32]) {
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
// swizzle): `next` bytes from one group of 64 columns to the next, 1024 bytes from one group of eight k to the next.
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(const void* smem_ptr, uint32_t next) {
  return (uint64_t)((smem_u32(smem_ptr) >> 4) & 0x3FFF) | (uint64_t)(next >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)2 << 61;
}

__global__ void __launch_bounds__(kMuThreads, 1)
mla_umma_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const MlaUmmaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem_raw);
  uint64_t* s_full = q_full + 2;      // [2] scores complete
  uint64_t* s_empty = q_full + 4;     // [2] scores read (an arrival per warp)
  uint64_t* p_full = q_full + 6;      // [2] probabilities written (an arrival per warp)
  uint64_t* pv_done = q_full + 8;     // [2] the tile's products are done: its probabilities are free, O is at rest
  uint64_t* k_full = q_full + 10;     // [kMuStages]
  uint64_t* k_empty = k_full + kMuStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(k_empty + kMuStages);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t base_u32 = smem_u32(smem_raw);
  uint8_t* q_s = smem_raw + 1024 + ((1024 - ((base_u32 + 1024) & 1023)) & 1023);
  uint8_t* k_s = q_s + (size_t)(kMuBoxes - kMuQTmem) * kMuQBox;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = blockIdx.x & 1, split = blockIdx.x >> 1, hg = blockIdx.y, b = blockIdx.z;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1 + 4);          // the copy of one part, the four warps that write the other
    for (int s = 0; s < kMuStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], 4);
      mbar_init(&p_full[s], 4);
      mbar_init(&pv_done[s], 1);
    }
    *failed = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();
  const int len = p.lens[b];
  const int k_begin = split * p.chunk, k_end = min(len, k_begin + p.chunk);
  const int n = k_end > k_begin ? (k_end - k_begin + kMuTile - 1) / kMuTile : 0;
  const int tail = n ? k_end - k_begin - (n - 1) * kMuTile : kMuTile;      // positions of the last tile
  auto give_up = [&](int code) {
    *failed = 1;
    atomicCAS(p.err, 0, code);
  };

  if (warp == 0) {
    const int whole = tail < kMuTile ? n - 1 : n;
    if (lane == 0 && n) {
      mbar_arrive_expect_tx(q_full, (kMuBoxes - kMuQTmem) * kMuQBox);
      for (int i = kMuQTmem; i < kMuBoxes; ++i)
        tma_load_2d(q_s + (size_t)(i - kMuQTmem) * kMuQBox, &q_map, 64 * i, b * p.n_heads + 128 * hg, q_full);
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < whole && !*failed; ++i) {
        if (!mbar_wait_spin(&k_empty[s], ph ^ 1u)) { give_up(DERR_EMPTY_WAIT); break; }
        mbar_arrive_expect_tx(&k_full[s], kMuStage);
        mu_load_4d(k_s + (size_t)s * kMuStage, &k_map, 0, k_begin + i * kMuTile, 0, b, &k_full[s]);   // all nine groups of 64 columns
        if (++s == kMuStages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    __syncwarp();
    if (whole < n) {
      // a last tile of `tail` rows: what the cache holds behind them may not be memory, and would not stay out of the products
      // (0 x NaN is NaN)
      const int s = whole % kMuStages;
      const bool ok = __all_sync(0xffffffffu, !*failed && mbar_wait_spin(&k_empty[s], ((whole / kMuStages) & 1) ^ 1u));
      if (ok) {
        const __nv_bfloat16* src = p.cache + (size_t)b * p.seq_stride + (size_t)(k_begin + whole * kMuTile) * kMuRow;
        const uint32_t dst = smem_u32(k_s + (size_t)s * kMuStage);
#pragma unroll 4
        for (int j = lane; j < kMuTile * kMuBoxes * 8; j += 32) {                    // pieces of 16 bytes
          const int r = j / (kMuBoxes * 8), c = j - r * (kMuBoxes * 8);
          const uint32_t at = dst + (uint32_t)((c >> 3) * kMuKBox + r * 128 + (((c & 7) ^ (r & 7)) << 4));
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(src + (r < tail ? r * kMuRow + 8 * c : 0)), "r"(r < tail ? 16u : 0u) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&k_full[s]);
      } else {
        give_up(DERR_EMPTY_WAIT);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t idesc_s = umma_idesc_bf16(kMuTile), idesc_o = umma_idesc_bf16(kMuHalf) | (1u << 16);   // (bit 16: B is N-major)
    const uint64_t qd = umma_desc_sw128(q_s), kd = umma_desc_sw128(k_s);
    const uint64_t vd = umma_desc_sw128_mn(k_s + (size_t)(half * 4) * kMuKBox, kMuKBox);
    bool ok = n == 0 || mbar_wait_spin(q_full, 0);
    int ks = 0, vs = 0;                  // stages of the tiles whose scores / products come next
    uint32_t kph = 0;
    for (int i = 0; i <= n && ok && n; ++i) {
      if (i < n) {
        const int s = i & 1;
        ok = mbar_wait_spin(&k_full[ks], kph) && mbar_wait_spin(&s_empty[s], ((i >> 1) & 1) ^ 1u);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint32_t d = tmem + (uint32_t)(kMuColS + s * kMuTile);
#pragma unroll 1
          for (int c = 0; c < kMuBoxes; ++c) {
            const uint64_t bd = kd + (uint64_t)((ks * kMuStage + c * kMuKBox) >> 4);
            if (c < kMuQTmem) {
              const uint32_t a_t = tmem + (uint32_t)(kMuColQ + 32 * c);
#pragma unroll
              for (int k16 = 0; k16 < 4; ++k16) umma_f16_ts(d, a_t + 8u * k16, bd + 2 * k16, idesc_s, (c | k16) != 0);
            } else {
              const uint64_t ad = qd + (uint64_t)((c - kMuQTmem) * (kMuQBox >> 4));
#pragma unroll
              for (int k16 = 0; k16 < 4; ++k16) umma_f16(d, ad + 2 * k16, bd + 2 * k16, idesc_s, 1u);
            }
          }
          umma_commit(&s_full[s]);
        }
        __syncwarp();
        if (++ks == kMuStages) {
          ks = 0;
          kph ^= 1u;
        }
      }
      if (i > 0) {
        const int t = i - 1, st = t & 1;
        ok = mbar_wait_spin(&p_full[st], (t >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint64_t bd = vd + (uint64_t)((vs * kMuStage) >> 4);
#pragma unroll
          for (int term = 0; term < 2; ++term)
#pragma unroll
            for (int k = 0; k < kMuTile / 16; ++k)
              umma_f16_ts(tmem, tmem + (uint32_t)(kMuColP + st * kMuTile + 16 * term + 8 * k), bd + (uint64_t)(k * (2048 >> 4)), idesc_o,
                          t != 0 || term != 0 || k != 0);
          umma_commit(&pv_done[st]);
          umma_commit(&k_empty[vs]);
        }
        __syncwarp();
        if (++vs == kMuStages) vs = 0;
      }
    }
    if (!ok) give_up(DERR_FULL_WAIT);
  } else if (warp >= kMuFirstSoft) {
    const int q = warp & 3, head = 128 * hg + 32 * q + lane;
    const uint32_t t_lane = tmem + ((uint32_t)(32 * q) << 16);
    if (n) {
      // this head's first 256 latent queries as the A operand in tensor memory (rows behind the last head repeat it)
      const uint4* src = reinterpret_cast<const uint4*>(p.q + ((size_t)b * p.n_heads + min(head, p.n_heads - 1)) * kMuRow);
#pragma unroll 2
      for (int c = 0; c < kMuQTmem * 2; ++c) {
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 x = src[4 * c + j];
          r[4 * j] = x.x; r[4 * j + 1] = x.y; r[4 * j + 2] = x.z; r[4 * j + 3] = x.w;
        }
        tmem_st16(t_lane + (uint32_t)(kMuColQ + 16 * c), r);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    float m = -FLT_MAX, l = 0.f;       // reference of the exponentials (log2 units) and the row sum
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < n && ok; ++i) {
      const int s = i & 1;
      ok = __all_sync(0xffffffffu, mbar_wait_spin(&s_full[s], (i >> 1) & 1));
      if (!ok) break;
      tc_fence_after();
      float v[32];
      mu_ld32(t_lane + (uint32_t)(kMuColS + s * kMuTile), v);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[s]);
      const int valid = i == n - 1 ? tail : kMuTile;
      float mx = -FLT_MAX;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        v[j] = j < valid ? v[j] * p.scale : -FLT_MAX;
        mx = fmaxf(mx, v[j]);
      }
      if (i == 0) m = mx;
      const bool grown = mx > m + kMuGrow;
      if (__any_sync(0xffffffffu, grown)) {
        const float m_new = grown ? mx : m, f = exp2f(m - m_new);
        ok = __all_sync(0xffffffffu, mbar_wait_spin(&pv_done[(i - 1) & 1], ((i - 1) >> 1) & 1));   // (the first tile never comes here)
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < kMuHalf; c += 16) {
          float o[16];
          tmem_ld16(t_lane + (uint32_t)c, o);
          uint32_t r[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(o[j] * f);
          tmem_st16(t_lane + (uint32_t)c, r);
        }
        tmem_st_wait();
        l *= f;
        m = m_new;
      }
      uint32_t hi[16], lo[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float a = 2 * j < valid ? exp2f(v[2 * j] - m) : 0.f, c = 2 * j + 1 < valid ? exp2f(v[2 * j + 1] - m) : 0.f;
        l += a;
        l += c;
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, c);
        const __nv_bfloat162 r = __floats2bfloat162_rn(a - __low2float(h), c - __high2float(h));
        hi[j] = *reinterpret_cast<const uint32_t*>(&h);
        lo[j] = *reinterpret_cast<const uint32_t*>(&r);
      }
      if (i >= 2) {                    // the products of the tile before last have read their probabilities
        ok = __all_sync(0xffffffffu, mbar_wait_spin(&pv_done[s], ((i - 2) >> 1) & 1));
        if (!ok) break;
        tc_fence_after();
      }
      tmem_st16(t_lane + (uint32_t)(kMuColP + s * kMuTile), hi);
      tmem_st16(t_lane + (uint32_t)(kMuColP + s * kMuTile + 16), lo);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[s]);
    }
    if (ok && n) ok = __all_sync(0xffffffffu, mbar_wait_spin(&pv_done[(n - 1) & 1], ((n - 1) >> 1) & 1));
    if (!ok) give_up(DERR_TMEM);
    tc_fence_after();
    // ---- results: 32 rows x 32 columns at a time through shared memory (the stages are free), so that rows leave in whole lines
    float* turn = reinterpret_cast<float*>(k_s) + q * (32 * 33);
    const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll 1
    for (int c = 0; c < kMuHalf && ok; c += 32) {
      float o[32];
      if (n) {
        mu_ld32(t_lane + (uint32_t)c, o);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) turn[lane * 33 + j] = p.n_splits == 1 ? o[j] * inv : o[j];
      __syncwarp();
#pragma unroll 4
      for (int r = 0; r < 32; ++r) {
        const int hd = 128 * hg + 32 * q + r;
        if (hd >= p.n_heads) break;
        const size_t bh = (size_t)b * p.n_heads + hd;
        const float x = turn[r * 33 + lane];
        if (p.n_splits == 1) p.out[bh * kMuLat + half * kMuHalf + c + lane] = __float2bfloat16_rn(x);
        else p.part_o[(bh * p.n_splits + split) * kMuLat + half * kMuHalf + c + lane] = x;
      }
      __syncwarp();
    }
    if (ok && p.n_splits > 1 && half == 0 && head < p.n_heads) {
      float* ml = p.part_ml + (((size_t)b * p.n_heads + head) * p.n_splits + split) * 2;
      ml[0] = m;                       // (-FLT_MAX where the split has no positions)
      ml[1] = l;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*failed && threadIdx.x == 0) {
    // copies and products that are still in flight target this CTA's memories: give them time to land before leaving
    for (int i = 0; i < 10000; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// False: the call is for the other kernel.  The tensor map wants aligned sequences that lie one behind the other: views that
// overlap, and a stride that nobody reads because there is one sequence, stay with the kernel that forms its own addresses.
bool mla_umma_supported(const void* q, const void* cache, size_t n_heads, size_t seq_stride, size_t batch, size_t max_len) {
  return n_heads >= 64 && ((uintptr_t)q & 15) == 0 && ((uintptr_t)cache & 15) == 0 && seq_stride % 8 == 0 && seq_stride >= max_len * kMuRow && batch <= 65535 &&
         encode_tiled() != nullptr;
}

// The attention over one latent cache with `n_splits` splits of `chunk` positions each.
int launch_mla_umma(tq_ctx* ctx, const void* q, const void* cache, const int* lens, size_t batch, size_t n_heads, size_t seq_stride, size_t max_len,
                    float scale, int n_splits, int chunk, void* out, float* part_o, float* part_ml) {
  MlaUmmaParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.cache = static_cast<const __nv_bfloat16*>(cache);
  p.seq_stride = seq_stride;
  p.lens = lens;
  p.n_heads = (int)n_heads;
  p.n_splits = n_splits;
  p.chunk = chunk;
  p.scale = scale * 1.4426950408889634f;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.part_o = part_o;
  p.part_ml = part_ml;
  p.err = ctx->dev_err;
  CUtensorMap qm, km;
  const cuuint64_t gdim[4] = {64, (cuuint64_t)max_len, (cuuint64_t)kMuBoxes, (cuuint64_t)batch};
  const cuuint64_t gstride[3] = {(cuuint64_t)kMuRow * 2, 128, (cuuint64_t)seq_stride * 2};
  const cuuint32_t box[4] = {64, (cuuint32_t)kMuTile, (cuuint32_t)kMuBoxes, 1}, estr[4] = {1, 1, 1, 1};
  if (!encode_bf16_k64(&qm, q, batch * n_heads, kMuRow, kMuRow, 128) ||
      encode_tiled()(&km, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(cache), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return fail(ctx, TQ_ECUDA, "cuTensorMapEncodeTiled failed");
  TQ_CUDA(ctx, cudaFuncSetAttribute(mla_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMuSmem));
  TQ_CUDA(ctx, launch_k(ctx, mla_umma_kernel, dim3((unsigned)(2 * n_splits), (unsigned)((n_heads + 127) / 128), (unsigned)batch), dim3(kMuThreads),
                        kMuSmem, qm, km, p));
  return TQ_OK;
}

}  // namespace tq
