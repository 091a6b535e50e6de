// Differential attention of many rows on the 5th-generation tensor cores (see diff_attention.cuh; diff_attention.cu has the mma.sync kernels and
// the rule between them): bf16, maps of 64, values of 128; f32 scores, sums and outputs, probabilities in two bf16 terms, as there.
//
// The form of gqa_prefill_umma.cu with the two maps of 128 (position, head) pairs in the place of its two query tiles: a CTA ends up with a1 and a2
// of its rows in tensor memory and finishes the difference and the head norm itself.
//   warp 0        copies Q once, then K (a box per map) and V tiles of 128 keys
//   warps 1, 2    issue a map's MMAs: S = Q K^T, then O += (P_hi + P_lo) V
//   warp 3        zeroes the V rows behind the last key (where the values of a key that a row of the tiles does not see are not finite, that row is
//                 formed once more, over its own keys)
//   warps 4..7, 8..11   softmax of a map, a thread per row, the scores of a tile in registers: the two terms (64 columns each) take their place
// Only tiles with visible keys are visited: those of the kept first tokens, then those of the window.
// What bounds it: 2 x (4 + 16) MMAs of 128 x 128 x 16 a tile (about 3100 cycles) against 2 x 128 exponentials a thread (2050).  Prompts of 1024, 820,
// 615 and 410 tokens, 16 heads, 4 KV heads, window 512: 124 us a layer (mma.sync kernel) -> 75.
#include <cfloat>

#include <cuda_bf16.h>

#include "attn_umma.cuh"
#include "diff_attention.cuh"

namespace tq {

constexpr int kDuaThreads = 384, kDuaStages = 3, kDuaV = 128;
constexpr int kDuaStage = 4 * kPfBox;                 // K of map 1, of map 2, V in two halves
constexpr size_t kDuaSmem = 1024 + 1024 + 2 * (size_t)kPfBox + kDuaStages * (size_t)kDuaStage;

struct DiffUmmaParams {
  DiffAttn a;
  RaggedBatch b;
  int group;
  const __nv_bfloat16 *q, *k, *v;
  __nv_bfloat16* out;
  long long ldq, ldo;
  int* err;
};

__global__ void __launch_bounds__(kDuaThreads, 1)
diff_attention_umma_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                           const __grid_constant__ DiffUmmaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem_raw);
  uint64_t* k_full = q_full + 1;                      // [stages]
  uint64_t* v_full = k_full + kDuaStages;
  uint64_t* kv_empty = v_full + kDuaStages;           // [stages] both maps' products done
  uint64_t* v_raw = kv_empty + kDuaStages;            // the last tile's V, before the rows behind the last key are zeroed
  uint64_t* s_full = v_raw + 1;                       // [map]
  uint64_t* p_full = s_full + 2;
  uint64_t* o_done = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);   // a map's softmax gave up
  uint8_t* q_s = smem_raw + 1024 + ((1024 - ((smem_u32(smem_raw) + 1024) & 1023)) & 1023);
  uint8_t* kv_s = q_s + 2 * kPfBox;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  pdl_launch_dependents();
  const int kvh = blockIdx.y, sq = blockIdx.z;
  const int row0 = p.b.seq_rows ? p.b.seq_rows[sq] : sq, n_q = p.b.seq_rows ? p.b.seq_rows[sq + 1] - row0 : 1;
  const int ppt = kPfTile / p.group;
  const int i0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * ppt;       // first query of this CTA; the last see the most keys and go first
  if (i0 >= n_q || row0 < 0 || row0 + n_q > p.b.rows) return;
  const int i1 = min(i0 + ppt, n_q) - 1;
  const int p0 = p.b.row_pos[row0 + i0], p1 = p0 + (i1 - i0);
  const int crow = p.b.cache_row[row0 + i0];
  // every row of the range has to be in the cache (the embedding kernel has reported one that is not)
  if (!(crow >= p0 && p.b.cache_row[row0 + i1] == crow + (i1 - i0) && (size_t)(crow + (i1 - i0)) < p.b.cache_rows)) return;
  const int seq0 = crow - p0;                         // cache row of the sequence's position 0
  // visible key tiles: the kept tokens' tiles that lie before the window's, then the window's
  const int lo_t = max(0, p0 - p.a.window + 1) / kPfTile, hi_t = p1 / kPfTile;
  const int n_kept = min((min(p.a.keep_first, p1 + 1) + kPfTile - 1) / kPfTile, lo_t);
  const int n = n_kept + hi_t - lo_t + 1, valid = p1 + 1 - hi_t * kPfTile;   // tiles; keys of the last
  auto key_of = [&](int i) { return (i < n_kept ? i : lo_t + i - n_kept) * kPfTile; };

  if (warp == 0) {
    if (lane == 0) {
      mbar_init(q_full, 1);
      for (int s = 0; s < kDuaStages; ++s) {
        mbar_init(&k_full[s], 1);
        mbar_init(&v_full[s], 1);
        mbar_init(&kv_empty[s], 2);
      }
      mbar_init(v_raw, 1);
      for (int x = 0; x < 2; ++x) {
        mbar_init(&s_full[x], 1);
        mbar_init(&p_full[x], 4);
        mbar_init(&o_done[x], 1);
      }
      *failed = 0;
      mbar_init_fence();
    }
  } else if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
  } else if (warp == 2 && lane == 0) {
    prefetch_map(&q_map);
    prefetch_map(&k_map);
    prefetch_map(&v_map);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto give_up = [&](int code) { atomicCAS(p.err, 0, code); };

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, 2u * kPfBox);
      for (int x = 0; x < 2; ++x) tma_load_3d(q_s + x * kPfBox, &q_map, 64 * x, kvh * p.group, row0 + i0, q_full);
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < n; ++i) {
        if (!mbar_wait_spin(&kv_empty[s], ph ^ 1u)) {
          give_up(DERR_EMPTY_WAIT);
          break;
        }
        uint8_t* at = kv_s + s * kDuaStage;
        const int row = seq0 + key_of(i);
        mbar_arrive_expect_tx(&k_full[s], 2u * kPfBox);
        for (int x = 0; x < 2; ++x) tma_load_3d(at + x * kPfBox, &k_map, kvh * 128 + 64 * x, row, 0, &k_full[s]);
        uint64_t* bar = i == n - 1 && valid < kPfTile ? v_raw : &v_full[s];
        mbar_arrive_expect_tx(bar, 2u * kPfBox);
        for (int c = 0; c < 2; ++c) tma_load_3d(at + (2 + c) * kPfBox, &v_map, kvh * kDuaV + 64 * c, row, 0, bar);
        if (++s == kDuaStages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    if (valid < kPfTile) {
      const int s = (n - 1) % kDuaStages;
      if (mbar_wait_spin(v_raw, 0)) {
        uint8_t* at = kv_s + s * kDuaStage + 2 * kPfBox;
        for (int i = lane; i < 2 * (kPfTile - valid) * 8; i += 32) {      // (a row's 128 bytes of either box, whatever their order)
          const int c = i & 7, row = valid + ((i >> 3) >> 1), box = (i >> 3) & 1;
          *reinterpret_cast<uint4*>(at + box * kPfBox + row * 128 + 16 * c) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&v_full[s]);
      } else {
        give_up(DERR_EMPTY_WAIT);
      }
    }
    __syncwarp();
  } else if (warp == 1 || warp == 2) {
    const bool leader = elect_one();
    const int x = warp - 1;
    const uint32_t idesc_s = umma_idesc_bf16(kPfTile), idesc_o = idesc_s | (1u << 16);   // (bit 16: B is N-major)
    const uint64_t qd = umma_desc_sw128(q_s + x * kPfBox), kd = umma_desc_sw128(kv_s + x * kPfBox), vd = pf_desc_mn(kv_s + 2 * kPfBox);
    const uint32_t s_t = tmem + (uint32_t)(x * 256), o_t = s_t + 128u;
    bool ok = mbar_wait_spin(q_full, 0);
    int st = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n && ok; ++i) {
      // (the scores' columns hold the probabilities of the tile before until its products are done)
      ok = mbar_wait_spin(&k_full[st], ph) && (i == 0 || mbar_wait_spin(&o_done[x], (i - 1) & 1));
      if (!ok) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_f16(s_t, qd + 2 * k, kd + (uint32_t)(st * (kDuaStage >> 4)) + 2 * k, idesc_s, k != 0);
        umma_commit(&s_full[x]);
      }
      __syncwarp();
      ok = mbar_wait_spin(&v_full[st], ph) && mbar_wait_spin(&p_full[x], i & 1);
      if (!ok) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int term = 0; term < 2; ++term)
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_f16_ts(o_t, s_t + 64u * term + 8u * k, vd + (uint32_t)(st * (kDuaStage >> 4)) + (uint32_t)(k * (2048 >> 4)), idesc_o, (i | term | k) != 0);
        umma_commit(&o_done[x]);
        umma_commit(&kv_empty[st]);
      }
      __syncwarp();
      if (++st == kDuaStages) {
        st = 0;
        ph ^= 1u;
      }
    }
    if (!ok) give_up(DERR_FULL_WAIT);
  } else {
    const int x = (warp - 4) >> 2, q4 = warp & 3, r = 32 * q4 + lane;
    const int qi = i0 + r / p.group, head = kvh * p.group + r % p.group;
    const bool live = qi <= i1;
    const int qpos = live ? p0 + (qi - i0) : -1;
    const float sl2 = p.a.scale * 1.44269504088896340736f;
    const uint32_t s_t = tmem + ((uint32_t)(32 * q4) << 16) + (uint32_t)(x * 256), o_t = s_t + 128u;
    float m = -FLT_MAX, l = 0.f;
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < n && ok; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait_spin(&s_full[x], i & 1));
      if (!ok) break;
      tc_fence_after();
      const int key0 = key_of(i);
      float v[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float u[32];
        pf_ld32(s_t + 32u * c, u);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[32 * c + j] = u[j];
      }
      // keys first .. last of the tile count, and those below keep
      const int last = qpos - key0, first = qpos - p.a.window + 1 - key0, keep = p.a.keep_first - key0;
      const bool whole = __all_sync(0xffffffffu, last >= kPfTile - 1 && (first <= 0 || keep >= kPfTile));
#pragma unroll
      for (int j = 0; j < kPfTile; ++j) v[j] *= sl2;
      if (!whole) {
#pragma unroll
        for (int j = 0; j < kPfTile; ++j) v[j] = j <= last && (j >= first || j < keep) ? v[j] : -INFINITY;
      }
      float mx = -FLT_MAX;
#pragma unroll
      for (int j = 0; j < kPfTile; ++j) mx = fmaxf(mx, v[j]);
      const bool grown = mx > m;
      if (i == 0) {
        m = mx;
      } else if (__any_sync(0xffffffffu, grown)) {    // (the products so far are done, or these scores would not be here)
        const float m_new = grown ? mx : m, f = ex2(m - m_new);
#pragma unroll 1
        for (int c = 0; c < kDuaV; c += 16) {
          float o[16];
          tmem_ld16(o_t + (uint32_t)c, o);
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) w[j] = __float_as_uint(o[j] * f);
          tmem_st16(o_t + (uint32_t)c, w);
        }
        l *= f;
        m = m_new;
      }
      const float base = m == -FLT_MAX ? 0.f : m;     // (nothing seen yet: every weight below becomes zero)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t hi[16], lo[16];
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float a = ex2(v[32 * c + 2 * j] - base), e = ex2(v[32 * c + 2 * j + 1] - base);
          sum[j & 3] += a + e;
          const __nv_bfloat162 h = __floats2bfloat162_rn(a, e);
          const __nv_bfloat162 d = __floats2bfloat162_rn(a - __low2float(h), e - __high2float(h));
          hi[j] = *reinterpret_cast<const uint32_t*>(&h);
          lo[j] = *reinterpret_cast<const uint32_t*>(&d);
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        tmem_st16(s_t + 16u * c, hi);
        tmem_st16(s_t + 64u + 16u * c, lo);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[x]);
    }
    // ---- both maps' outputs, a2 through shared memory.  The stages are free when both maps' products are done.  Each map's group looks at its
    // own map's barrier, since a wait for a parity is only sound for a thread that knows the phase before to be over (the scores of tile n - 1
    // stand behind this map's products of tile n - 2; the other map may be tiles behind), and the groups then meet.
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait_spin(&o_done[x], (n - 1) & 1));
    if (!ok) {
      give_up(DERR_TMEM);
      *failed = 1;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    ok = *failed == 0;
    tc_fence_after();
    float* a2 = reinterpret_cast<float*>(kv_s) + r;   // [column][row]
    if (ok && x == 1) {
      const float w2 = p.a.lambda / l;
#pragma unroll 1
      for (int c = 0; c < kDuaV; c += 32) {
        float o[32];
        pf_ld32(o_t + (uint32_t)c, o);
#pragma unroll
        for (int j = 0; j < 32; ++j) a2[(c + j) * kPfTile] = o[j] * w2;
      }
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (ok && x == 0) {
      const float w1 = 1.0f / l;
      float o[kDuaV], sqs = 0.f;
#pragma unroll
      for (int c = 0; c < kDuaV; c += 32) {
        float u[32];
        pf_ld32(o_t + (uint32_t)c, u);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          o[c + j] = u[j] * w1 - a2[(c + j) * kPfTile];
          sqs += o[c + j] * o[c + j];
        }
      }
      const float inv = p.a.out_scale / sqrtf(sqs / (float)kDuaV + p.a.eps);
      if (live) {
        uint4* y = reinterpret_cast<uint4*>(p.out + (size_t)(row0 + qi) * p.ldo + (size_t)head * kDuaV);
#pragma unroll
        for (int j = 0; j < kDuaV / 8; ++j) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(o[8 * j + 2 * e] * inv, o[8 * j + 2 * e + 1] * inv);
            w[e] = *reinterpret_cast<const uint32_t*>(&h);
          }
          y[j] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      unsigned rows = __ballot_sync(0xffffffffu, live && !(fabsf(sqs) <= FLT_MAX));
      const size_t ke = (size_t)p.a.kv_heads * 128, ve = (size_t)p.a.kv_heads * kDuaV;
      while (rows) {
        const int src = __ffs(rows) - 1;
        rows &= rows - 1;
        const int at = row0 + __shfl_sync(0xffffffffu, qi, src), pos = __shfl_sync(0xffffffffu, qpos, src), h = __shfl_sync(0xffffffffu, head, src);
        const int lo = max(0, pos - p.a.window + 1), kept = min(p.a.keep_first, lo);
        const __nv_bfloat16* vb = p.v + (size_t)seq0 * ve + (size_t)kvh * kDuaV;
        float sum[4] = {0.f, 0.f, 0.f, 0.f}, sq = 0.f;
#pragma unroll 1
        for (int mp = 0; mp < 2; ++mp) {
          const __nv_bfloat16* kb = p.k + (size_t)seq0 * ke + (size_t)kvh * 128 + 64 * mp;
          float qr[2], rm = -FLT_MAX, rl = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < 2; ++i) qr[i] = __bfloat162float(p.q[(size_t)at * p.ldq + (size_t)h * 128 + 64 * mp + 2 * lane + i]);
          attend_row(kb, ke, vb, ve, 0, kept, qr, sl2, lane, rm, rl, acc);
          attend_row(kb, ke, vb, ve, lo, pos + 1, qr, sl2, lane, rm, rl, acc);
#pragma unroll
          for (int i = 0; i < 4; ++i) sum[i] = mp ? sum[i] - acc[i] * (p.a.lambda / rl) : acc[i] * (1.0f / rl);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) sq += sum[i] * sum[i];
        const float rinv = p.a.out_scale / sqrtf(warp_sum(sq) / (float)kDuaV + p.a.eps);
#pragma unroll
        for (int i = 0; i < 4; ++i) p.out[(size_t)at * p.ldo + (size_t)h * kDuaV + 4 * lane + i] = __float2bfloat16_rn(sum[i] * rinv);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// The head sizes and alignments that the kernel is written for.
bool diff_attention_umma_supported(const DiffAttn& a, const RaggedBatch& b, const void* q, size_t ldq, const void* k, const void* v, const void* out, size_t ldo) {
  const int group = a.heads / a.kv_heads;
  return encode_tiled() && a.dim == 64 && a.dim_pad == 64 && a.vdim == kDuaV && a.vdim_pad == kDuaV && group <= kPfTile && kPfTile % group == 0 && ldq % 8 == 0 &&
         ldo % 8 == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) == 0 && b.cache_rows > 0 && b.cache_rows < (1u << 31);
}

int launch_diff_attention_umma(tq_ctx* ctx, const DiffAttn& a, const RaggedBatch& b, const void* q, size_t ldq, const void* k, const void* v, void* out,
                               size_t ldo) {
  DiffUmmaParams p;
  p.a = a;
  p.b = b;
  p.group = a.heads / a.kv_heads;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.ldq = (long long)ldq;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ldo = (long long)ldo;
  p.err = ctx->dev_err;
  const size_t ke = (size_t)a.kv_heads * 128, ve = (size_t)a.kv_heads * kDuaV;
  const int ppt = kPfTile / p.group;
  CUtensorMap qm, km, vm;
  if (!encode_bf16_boxes(&qm, q, 128, (size_t)a.heads, (size_t)b.rows, 256, ldq * 2, (unsigned)p.group, (unsigned)ppt) ||
      !encode_bf16_boxes(&km, k, ke, b.cache_rows, 1, ke * 2, ke * 2 * b.cache_rows, kPfTile, 1) ||
      !encode_bf16_boxes(&vm, v, ve, b.cache_rows, 1, ve * 2, ve * 2 * b.cache_rows, kPfTile, 1))
    return fail(ctx, TQ_ECUDA, "cuTensorMapEncodeTiled failed");
  TQ_CUDA(ctx, cudaFuncSetAttribute(diff_attention_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDuaSmem));
  TQ_CUDA(ctx, launch_k(ctx, diff_attention_umma_kernel, dim3((unsigned)((b.max_q + ppt - 1) / ppt), (unsigned)a.kv_heads, (unsigned)b.n_seqs),
                        dim3(kDuaThreads), kDuaSmem, qm, km, vm, p));
  return TQ_OK;
}

}  // namespace tq
