// Causal attention of a chunk of new positions on the 5th-generation tensor cores (attention.cu has the interface, the mma.sync kernel
// and the rule between the two): bf16 q / K / V, f32 scores and sums, bf16 probabilities, as there.
//
// A CTA takes two query tiles of 128 rows (128 / group positions x the group's heads of one KV head) over the same key tiles of 128:
//   warp 0        copies Q once, then K and V tiles (two stages)
//   warps 1, 2    issue a query tile's MMAs: S = Q K^T (both from shared memory), then O += P V (P from tensor memory, V N-major)
//   warp 3        zeroes the V rows behind the last key (whatever the cache holds there must not meet a probability of zero; where the values of a
//                 later key of the chunk are not finite, the rows before it are formed once more, over their own keys)
//   warps 4..7, 8..11   softmax of a query tile, a thread per row: maximum, probabilities over the scores' columns, and, only where a
//                 row's maximum grew, a rescaling of O (a reference that may lag behind the maximum would save a tenth of the time, but
//                 then the largest probability is no longer 1, which bf16 holds exactly: errors against 64 bits 1.50e-3 -> 1.65e-3)
// Tensor memory: S / P and O of both tiles, 4 x 128 columns.  While one tile's scores are turned into probabilities, the other tile's
// products run.  What bounds it: per pair of tiles 16 + 16 MMAs of 128 x 128 x 16 (about 2700 cycles) against 2 x 128 exponentials a
// thread (2050 cycles of a scheduler's pipe).  32 heads, 8 KV heads, us (mma.sync kernel -> this): 2048 positions 221 -> 88 (390 TFLOP/s),
// 2 x 1000 behind 777 cached ones 248 -> 94, 512 positions 26.7 -> 19.2.
#include <cfloat>

#include <cuda_bf16.h>

#include "attn_umma.cuh"
#include "internal.h"

namespace tq {

constexpr int kPfThreads = 384, kPfHd = 128;
constexpr int kPfStage = 4 * kPfBox;                  // K, V: two boxes each
constexpr int kPfStages = 2;
constexpr size_t kPfSmem = 1024 + 1024 + 4 * (size_t)kPfBox + kPfStages * (size_t)kPfStage;

struct PrefillUmmaParams {
  const int* cache_start;
  int q_len, n_heads, n_kv, group, rows_max;          // rows_max: positions that a sequence's cache holds
  float scale_log2;
  const __nv_bfloat16 *q, *k, *v;
  size_t seq_stride;
  void* out;
  int out_f32;
  int* err;
};

__global__ void __launch_bounds__(kPfThreads, 1)
gqa_prefill_umma_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                        const __grid_constant__ PrefillUmmaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem_raw);
  uint64_t* k_full = q_full + 1;                      // [stages]
  uint64_t* v_full = k_full + kPfStages;
  uint64_t* kv_empty = v_full + kPfStages;            // [stages] both query tiles' products done
  uint64_t* v_raw = kv_empty + kPfStages;             // the last tile's V, before the rows behind the last key are zeroed
  uint64_t* s_full = v_raw + 1;                       // [query tile]
  uint64_t* p_full = s_full + 2;
  uint64_t* o_done = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  uint8_t* q_s = smem_raw + 1024 + ((1024 - ((smem_u32(smem_raw) + 1024) & 1023)) & 1023);
  uint8_t* kv_s = q_s + 4 * kPfBox;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.y, b = blockIdx.z;
  const int ppt = kPfTile / p.group, pos0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * 2 * ppt;   // (the longest rows first)
  if (warp == 0) {
    if (lane == 0) {
      mbar_init(q_full, 1);
      for (int s = 0; s < kPfStages; ++s) {
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
  pdl_wait();
  pdl_launch_dependents();
  auto give_up = [&](int code) { atomicCAS(p.err, 0, code); };
  const int start = p.cache_start[b];
  // The chunk must lie inside the sequence's cache rows (cache_start comes from device memory): if not, nothing is read or written
  // for this sequence and the status word says why.
  const bool inside = start >= 0 && (long long)start + p.q_len <= p.rows_max;
  if (!inside && threadIdx.x == 0 && blockIdx.x == 0 && kvh == 0) give_up(DERR_POSITION);
  const int k_end = inside ? start + min(p.q_len, pos0 + 2 * ppt) : 0;
  const int n = (k_end + kPfTile - 1) / kPfTile, valid = k_end - (n - 1) * kPfTile;      // key tiles; keys of the last

  if (warp == 0) {
    if (lane == 0 && n > 0) {
      mbar_arrive_expect_tx(q_full, 4u * kPfBox);
      for (int x = 0; x < 2; ++x)
        for (int c = 0; c < 2; ++c)
          tma_load_3d(q_s + (2 * x + c) * kPfBox, &q_map, 64 * c, kvh * p.group, b * p.q_len + pos0 + x * ppt, q_full);
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < n; ++i) {
        if (!mbar_wait_spin(&kv_empty[s], ph ^ 1u)) {
          give_up(DERR_EMPTY_WAIT);
          break;
        }
        uint8_t* at = kv_s + s * kPfStage;
        mbar_arrive_expect_tx(&k_full[s], 2u * kPfBox);
        for (int c = 0; c < 2; ++c) tma_load_3d(at + c * kPfBox, &k_map, kvh * kPfHd + 64 * c, i * kPfTile, b, &k_full[s]);
        uint64_t* bar = i == n - 1 && valid < kPfTile ? v_raw : &v_full[s];
        mbar_arrive_expect_tx(bar, 2u * kPfBox);
        for (int c = 0; c < 2; ++c) tma_load_3d(at + (2 + c) * kPfBox, &v_map, kvh * kPfHd + 64 * c, i * kPfTile, b, bar);
        if (++s == kPfStages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    if (n > 0 && valid < kPfTile) {
      const int s = (n - 1) % kPfStages;
      if (mbar_wait_spin(v_raw, 0)) {
        uint8_t* at = kv_s + s * kPfStage + 2 * kPfBox;
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
    const uint64_t qd = umma_desc_sw128(q_s + 2 * x * kPfBox), kd = umma_desc_sw128(kv_s), vd = pf_desc_mn(kv_s + 2 * kPfBox);
    const uint32_t s_t = tmem + (uint32_t)(x * 256), o_t = s_t + 128u;
    bool ok = n == 0 || mbar_wait_spin(q_full, 0);
    int st = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n && ok; ++i) {
      // (the scores' columns hold the probabilities of the tile before until its products are done)
      ok = mbar_wait_spin(&k_full[st], ph) && (i == 0 || mbar_wait_spin(&o_done[x], (i - 1) & 1));
      if (!ok) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = (uint32_t)((k >> 2) * (kPfBox >> 4) + 2 * (k & 3));
          umma_f16(s_t, qd + off, kd + (uint32_t)(st * (kPfStage >> 4)) + off, idesc_s, k != 0);
        }
        umma_commit(&s_full[x]);
      }
      __syncwarp();
      ok = mbar_wait_spin(&v_full[st], ph) && mbar_wait_spin(&p_full[x], i & 1);
      if (!ok) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16_ts(o_t, s_t + 8u * k, vd + (uint32_t)(st * (kPfStage >> 4)) + (uint32_t)(k * (2048 >> 4)), idesc_o, (i | k) != 0);
        umma_commit(&o_done[x]);
        umma_commit(&kv_empty[st]);
      }
      __syncwarp();
      if (++st == kPfStages) {
        st = 0;
        ph ^= 1u;
      }
    }
    if (!ok) give_up(DERR_FULL_WAIT);
  } else {
    const int x = (warp - 4) >> 2, q4 = warp & 3, r = 32 * q4 + lane;
    const int pos = pos0 + x * ppt + r / p.group, head = kvh * p.group + r % p.group;
    const bool live = pos < p.q_len;
    const int limit = live ? start + pos : -1;        // the last key of this row
    const uint32_t s_t = tmem + ((uint32_t)(32 * q4) << 16) + (uint32_t)(x * 256), o_t = s_t + 128u;
    float m = -FLT_MAX, l = 0.f;
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < n && ok; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait_spin(&s_full[x], i & 1));
      if (!ok) break;
      tc_fence_after();
      const int last = limit - i * kPfTile;           // keys 0 .. last of the tile count
      const bool whole = __all_sync(0xffffffffu, last >= kPfTile - 1);
      float mx = -FLT_MAX;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float v[32];
        pf_ld32(s_t + 32u * c, v);
        if (whole) {
#pragma unroll
          for (int j = 0; j < 32; ++j) mx = fmaxf(mx, v[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) mx = fmaxf(mx, 32 * c + j <= last ? v[j] : -FLT_MAX);
        }
      }
      mx = mx == -FLT_MAX ? mx : mx * p.scale_log2;
      if (i == 0) m = mx;
      const bool grown = mx > m;
      if (__any_sync(0xffffffffu, grown)) {           // (never in the first tile; the products so far are done, or these scores would not be here)
        const float m_new = grown ? mx : m, f = ex2(m - m_new);
#pragma unroll 1
        for (int c = 0; c < kPfHd; c += 32) {
          float o[32];
          pf_ld32(o_t + (uint32_t)c, o);
          uint32_t w0[16], w1[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            w0[j] = __float_as_uint(o[j] * f);
            w1[j] = __float_as_uint(o[16 + j] * f);
          }
          tmem_st16(o_t + (uint32_t)c, w0);
          tmem_st16(o_t + (uint32_t)c + 16u, w1);
        }
        l *= f;
        m = m_new;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float v[32];
        pf_ld32(s_t + 32u * c, v);
        if (whole) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = ex2(fmaf(v[j], p.scale_log2, -m));
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 32 * c + j <= last ? ex2(fmaf(v[j], p.scale_log2, -m)) : 0.f;
        }
        uint32_t w[16];
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          sum[j & 3] += v[2 * j] + v[2 * j + 1];
          const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          w[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        tmem_st16(s_t + 16u * c, w);                  // over scores that this thread has read
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[x]);
    }
    if (ok && n) ok = __all_sync(0xffffffffu, mbar_wait_spin(&o_done[x], (n - 1) & 1));
    if (!ok) give_up(DERR_TMEM);
    tc_fence_after();
    if (ok && n) {
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      const size_t at = (((size_t)b * p.q_len + (live ? pos : 0)) * p.n_heads + head) * kPfHd;
      float zero = 0.f;                               // NaN if some sum is not finite
#pragma unroll 1
      for (int c = 0; c < kPfHd; c += 32) {
        float o[32];
        pf_ld32(o_t + (uint32_t)c, o);
        if (!live) continue;
#pragma unroll
        for (int j = 0; j < 32; ++j) zero = fmaf(o[j], 0.f, zero);
        if (p.out_f32) {
          float4* y = reinterpret_cast<float4*>(static_cast<float*>(p.out) + at + c);
#pragma unroll
          for (int j = 0; j < 8; ++j) y[j] = make_float4(o[4 * j] * inv, o[4 * j + 1] * inv, o[4 * j + 2] * inv, o[4 * j + 3] * inv);
        } else {
          uint4* y = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + at + c);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(o[8 * j + 2 * e] * inv, o[8 * j + 2 * e + 1] * inv);
              w[e] = *reinterpret_cast<const uint32_t*>(&h);
            }
            y[j] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      unsigned rows = __ballot_sync(0xffffffffu, live && zero != zero);
      if (rows) {
        // Keys that rows of this CTA do not see and their tiles hold: from its first position on.
        const size_t ld = (size_t)p.n_kv * kPfHd;
        const __nv_bfloat16 *kb = p.k + (size_t)b * p.seq_stride + (size_t)kvh * kPfHd, *vb = p.v + (size_t)b * p.seq_stride + (size_t)kvh * kPfHd;
        float z = 0.f;
        for (int key = start + pos0 + 1; key < k_end; ++key)
#pragma unroll
          for (int i = 0; i < 4; ++i) z = fmaf(__bfloat162float(vb[(size_t)key * ld + 4 * lane + i]), 0.f, z);
        if (!__any_sync(0xffffffffu, z != z)) rows = 0u;
        while (rows) {
          const int src = __ffs(rows) - 1;
          rows &= rows - 1;
          const int row_limit = __shfl_sync(0xffffffffu, limit, src);
          const size_t row_at = __shfl_sync(0xffffffffu, (unsigned long long)at, src) + 4 * lane;
          float qr[4], rm = -FLT_MAX, rl = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < 4; ++i) qr[i] = __bfloat162float(p.q[row_at + i]);
          attend_row(kb, ld, vb, ld, 0, row_limit + 1, qr, p.scale_log2, lane, rm, rl, acc);
          const float rinv = rl > 0.f ? 1.0f / rl : 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (p.out_f32) static_cast<float*>(p.out)[row_at + i] = acc[i] * rinv;
            else static_cast<__nv_bfloat16*>(p.out)[row_at + i] = __float2bfloat16_rn(acc[i] * rinv);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

bool gqa_prefill_umma_supported(const void* q, const void* k, const void* v, const void* out, size_t seq_stride) {
  return encode_tiled() && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) == 0 && seq_stride % 8 == 0;
}

int launch_gqa_prefill_umma(tq_ctx* ctx, const void* q, const void* k, const void* v, const int* cache_start, size_t batch, size_t q_len,
                            size_t n_heads, size_t n_kv, size_t seq_stride, float scale, void* out, int out_f32) {
  const size_t group = n_heads / n_kv, row = n_kv * kPfHd, rows_max = seq_stride / row, per_cta = 2 * (kPfTile / group);
  PrefillUmmaParams p;
  p.cache_start = cache_start;
  p.q_len = (int)q_len;
  p.n_heads = (int)n_heads;
  p.n_kv = (int)n_kv;
  p.group = (int)group;
  p.rows_max = (int)rows_max;
  p.scale_log2 = scale * 1.44269504088896340736f;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k = static_cast<const __nv_bfloat16*>(k);
  p.v = static_cast<const __nv_bfloat16*>(v);
  p.seq_stride = seq_stride;
  p.out = out;
  p.out_f32 = out_f32;
  p.err = ctx->dev_err;
  CUtensorMap qm, km, vm;
  if (!encode_bf16_boxes(&qm, q, kPfHd, n_heads, batch * q_len, kPfHd * 2, n_heads * kPfHd * 2, (unsigned)group, (unsigned)(kPfTile / group)) ||
      !encode_bf16_boxes(&km, k, row, rows_max, batch, row * 2, seq_stride * 2, kPfTile, 1) || !encode_bf16_boxes(&vm, v, row, rows_max, batch, row * 2, seq_stride * 2, kPfTile, 1))
    return fail(ctx, TQ_ECUDA, "cuTensorMapEncodeTiled failed");
  TQ_CUDA(ctx, cudaFuncSetAttribute(gqa_prefill_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPfSmem));
  TQ_CUDA(ctx, launch_k(ctx, gqa_prefill_umma_kernel, dim3((unsigned)((q_len + per_cta - 1) / per_cta), (unsigned)n_kv, (unsigned)batch), dim3(kPfThreads),
                        kPfSmem, qm, km, vm, p));
  return TQ_OK;
}

}  // namespace tq
