// Kernels behind the reference's existing operator signatures.
//
//   sphkv_pool_decode         fused_decode.sphkv_decode        (fused_decode.py:12-26)
//   sphkv_pool_encode_append  fused_decode.sphkv_encode_append (fused_decode.py:28-35)
//   sphkv_qlut_logits         new_fused_decode.sphkv_logits    (new_fused_decode.py:22-43)
//   sphkv_ragged_logits       fused_decode.fused_decode_ragged (call sites only:
//                             spherical_kv_pipeline.py:1109-1125, 1866-1870)
//
// They read the LayerPool layout (sphkv_lut.py:77-103): one byte per centroid index and
// per radius code, post-RoPE keys, single sequence.  The arithmetic of
// decode_kernel.cu:10-246 is kept (sentinel mask for zero logits, +1e-8 in the final
// division, running-max radius scale with in-place re-quantisation); the work split is
// new: one CTA serves all query heads of a KV head per page through a q.centroid look-up
// table instead of staging a 64 KiB codebook per (query head, page).
#include <algorithm>

#include "common.cuh"

namespace sphkv {

constexpr int kPoolThreads = 256;

// ---- pool decode: per (KV head, logical page) partial (m, l, acc) for each query head ----
// The q.centroid table depends only on (query head, tier), not on the page: a CTA builds the tables
// of the tiers its pages use, then `wpp` warps share a page: each takes page_size / wpp tokens --
// logits through the table, softmax statistics by shuffles, one pass over its V rows that feeds the
// accumulators of four query heads at a time -- and the wpp (m, l, acc) triples of the page are
// folded through shared memory.  wpp is the largest split that leaves a warp 16 tokens, so 128-token
// pages (33 of them per head at 4K) fill the GPU as 16-token pages do.  Bound: latency of the table
// build and of the V rows (a 4000-token, 8-head step reads 8 MB).  That step, append and reduction included:
// 61.5 us with a warp walking a whole page, 21.9 us so.
constexpr int kPoolWarps = kPoolThreads / 32;
constexpr int kMaxPageRounds = 4;  // rounds of pages per CTA: amortise the tables once the GPU is full

__global__ void __launch_bounds__(kPoolThreads) pool_page_kernel(
    const float* __restrict__ q_all, const float* __restrict__ cb_flat,
    const int* __restrict__ tier_G_arr, const int* __restrict__ tier_g_arr,
    const uint8_t* __restrict__ theta_codes, const uint8_t* __restrict__ radius_codes,
    const float* __restrict__ r_scales, const __half* __restrict__ v_pool,
    const int* __restrict__ block_table, const int* __restrict__ bits_table,
    float* __restrict__ partial_out, int num_q_heads, int kv_groups, int num_tiers, int max_blocks,
    int page_size, int dh, int G_max, int cb_max, int g_max, float sm_scale, int wpp, int rounds,
    int stage_bytes) {
  const int hkv = blockIdx.x, tid = threadIdx.x;
  const int hq0 = hkv * kv_groups;
  const int warp = tid >> 5, lane = tid & 31;
  const int seg = page_size / wpp;             // tokens of a warp
  const int at_once = kPoolWarps / wpp;        // pages the CTA works on at a time
  const int sub = warp % wpp, group = warp / wpp;

  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* sq = reinterpret_cast<float*>(smem_raw);                 // [kv_groups][dh]
  float* lut = sq + kv_groups * dh;                                // [num_tiers][kv_groups][G_max][cb_max]
  // an even number of floats: the accumulators of fold_all are stored in 8-byte pieces
  float* slog_all = lut + ((num_tiers * kv_groups * G_max * cb_max + 1) & ~1);  // [warps][kv_groups][seg]
  float* srs_all = slog_all + kPoolWarps * kv_groups * seg;        // [warps][G_max]
  float* fold_all = srs_all + kPoolWarps * G_max;                  // wpp > 1: [warps][kv_groups][dh + 2]
  float* slog = slog_all + warp * kv_groups * seg;
  float* srs = srs_all + warp * G_max;
  // stage_bytes > 0: this warp's tokens of a page -- V rows, centroid indices, radii -- travel to shared
  // memory asynchronously, the first page's while the tables are built
  uint8_t* stage = smem_raw + (((fold_all + (wpp > 1 ? kPoolWarps * kv_groups * (dh + 2) : 0)) - sq) * 4 + 15) / 16 * 16 +
                   warp * stage_bytes;
  const int v_bytes = seg * dh * 2, c_bytes = seg * G_max;
  float* fold = fold_all + warp * kv_groups * (dh + 2);
  __shared__ unsigned s_tiers;

  if (tid == 0) s_tiers = 0;
  griddep_wait();
  griddep_launch();
  const int pg0 = blockIdx.y * at_once * rounds;
  const int pg_end = min(max_blocks, pg0 + at_once * rounds);
  auto page_of = [&](int k) -> int {
    const int page_idx = pg0 + k * at_once + group;
    return k < rounds && page_idx < max_blocks ? block_table[hkv * max_blocks + page_idx] : -1;
  };
  auto issue_stage = [&](int phys) {
    if (stage_bytes == 0 || phys < 0) return;
    const int64_t tok0 = (int64_t)phys * page_size + sub * seg;
    const uint32_t dst = smem_u32(stage);
    const uint8_t* vs = reinterpret_cast<const uint8_t*>(v_pool + tok0 * dh);
    for (int i = lane * 16; i < c_bytes; i += 512) {
      cp_async_16(dst + v_bytes + i, theta_codes + tok0 * G_max + i);
      cp_async_16(dst + v_bytes + c_bytes + i, radius_codes + tok0 * G_max + i);
    }
    for (int i = lane * 16; i < v_bytes; i += 512) cp_async_16(dst + i, vs + i);
    cp_async_commit();
  };
  int phys_next = page_of(0);
  issue_stage(phys_next);
  for (int i = tid; i < kv_groups * dh; i += blockDim.x) sq[i] = q_all[(int64_t)hq0 * dh + i];
  __syncthreads();
  for (int i = pg0 + tid; i < pg_end; i += blockDim.x)
    if (block_table[hkv * max_blocks + i] >= 0) atomicOr(&s_tiers, 1u << (bits_table[hkv * max_blocks + i] & 31));
  __syncthreads();
  // q . centroid tables; same summation order as decode_kernel.cu:186-188.  Groups of 16 and 32: a thread dots one
  // centroid row with every query head, so the row is read once.
  const unsigned tiers = s_tiers;
  const bool vec4 = (g_max & 3) == 0 && (dh & 3) == 0 && (reinterpret_cast<uintptr_t>(cb_flat) & 15) == 0;
  for (int ti = 0; ti < num_tiers; ++ti) {
    if (ti < 32 && !((tiers >> ti) & 1)) continue;
    const int G = tier_G_arr[ti], g = tier_g_arr[ti];
    const float* cb_t = cb_flat + ((int64_t)hkv * num_tiers + ti) * G_max * cb_max * g_max;
    float* lt = lut + (int64_t)ti * kv_groups * G_max * cb_max;
    if (vec4 && (g == 16 || g == 32)) {
      for (int i = tid; i < G * cb_max; i += blockDim.x) {
        const int c = i % cb_max, gg = i / cb_max;
        const float* cw = cb_t + ((int64_t)gg * cb_max + c) * g_max;
        float4 w4[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) w4[e] = __ldg(reinterpret_cast<const float4*>(cw) + e);
        if (g == 32) {
#pragma unroll
          for (int e = 4; e < 8; ++e) w4[e] = __ldg(reinterpret_cast<const float4*>(cw) + e);
        }
        for (int h = 0; h < kv_groups; ++h) {
          const float4* qg = reinterpret_cast<const float4*>(sq + h * dh + gg * g);
          float dot = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (e < 4 || g == 32) {
              const float4 q4 = qg[e];
              dot += q4.x * w4[e].x;
              dot += q4.y * w4[e].y;
              dot += q4.z * w4[e].z;
              dot += q4.w * w4[e].w;
            }
          }
          lt[(h * G_max + gg) * cb_max + c] = dot;
        }
      }
    } else {  // other group sizes: a thread per (query head, centroid), 16-byte pieces where rows allow it
      const bool pieces = vec4 && (g & 3) == 0;
      for (int i = tid; i < kv_groups * G * cb_max; i += blockDim.x) {
        const int c = i % cb_max, gg = (i / cb_max) % G, h = i / (cb_max * G);
        const float* qg = sq + h * dh + gg * g;
        const float* cw = cb_t + ((int64_t)gg * cb_max + c) * g_max;
        float dot = 0.f;
        if (pieces) {
          for (int d = 0; d < g; d += 4) {
            const float4 w = __ldg(reinterpret_cast<const float4*>(cw + d));
            dot += qg[d] * w.x;
            dot += qg[d + 1] * w.y;
            dot += qg[d + 2] * w.z;
            dot += qg[d + 3] * w.w;
          }
        } else {
          for (int d = 0; d < g; ++d) dot += qg[d] * cw[d];
        }
        lt[(h * G_max + gg) * cb_max + c] = dot;
      }
    }
  }
  __syncthreads();

  for (int k = 0; k < rounds; ++k) {
    const int page_idx = pg0 + k * at_once + group;
    const int phys = phys_next;
    phys_next = page_of(k + 1);
    if (page_idx < max_blocks && phys < 0 && sub == 0) {
      for (int h = 0; h < kv_groups; ++h) {
        float* po = partial_out + ((int64_t)(hq0 + h) * max_blocks + page_idx) * (dh + 2);
        if (lane == 0) { po[0] = -INFINITY; po[1] = 0.f; }
        for (int d = lane; d < dh; d += 32) po[2 + d] = 0.f;
      }
    }
    if (phys >= 0) {
      const int tier_idx = bits_table[hkv * max_blocks + page_idx];
      const int G = tier_G_arr[tier_idx];
      const float* lt = lut + (int64_t)tier_idx * kv_groups * G_max * cb_max;
      const int64_t tok0 = (int64_t)phys * page_size + sub * seg;
      __syncwarp();  // the previous page's readers of slog / srs are done
      for (int i = lane; i < G_max; i += 32) srs[i] = r_scales[(int64_t)phys * G_max + i];
      const bool staged = stage_bytes > 0;
      const uint8_t* th_rows = staged ? stage + v_bytes : theta_codes + tok0 * G_max;
      const uint8_t* rc_rows = staged ? stage + v_bytes + c_bytes : radius_codes + tok0 * G_max;
      const __half* v_rows = staged ? reinterpret_cast<const __half*>(stage) : v_pool + tok0 * dh;
      cp_async_wait<0>();
      __syncwarp();
      // logits: lane = (token, query head) pairs.  A byte becomes a float by planting it in the
      // mantissa of 2^23 (exact, and keeps the conversion off the special-function pipe).
      const bool words = (G_max & 3) == 0;
      for (int i = lane; i < seg * kv_groups; i += 32) {
        const int t = i % seg, h = i / seg;
        const uint8_t* th = th_rows + t * G_max;
        const uint8_t* rc = rc_rows + t * G_max;
        const float* lh = lt + (int64_t)h * G_max * cb_max;
        float logit_sum = 0.f;
        if (words) {
          for (int g0 = 0; g0 < G; g0 += 4) {
            const uint32_t tw = *reinterpret_cast<const uint32_t*>(th + g0);
            const uint32_t rw = *reinterpret_cast<const uint32_t*>(rc + g0);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (g0 + e < G) {
                const float rf = __uint_as_float(0x4B000000u | ((rw >> (8 * e)) & 0xFFu)) - 8388608.0f;
                const float r_hat = srs[g0 + e] * rf / 255.0f;
                logit_sum += r_hat * lh[(g0 + e) * cb_max + ((tw >> (8 * e)) & 0xFFu)];
              }
            }
          }
        } else {
          for (int gg = 0; gg < G; ++gg) {
            const float r_hat = srs[gg] * (float)rc[gg] / 255.0f;
            logit_sum += r_hat * lh[gg * cb_max + th[gg]];
          }
        }
        slog[h * seg + t] = (logit_sum == 0.f) ? -1e9f : logit_sum * sm_scale;
      }
      __syncwarp();
      // softmax statistics per head; the logits are replaced in place by exp(logit - max)
      for (int h = 0; h < kv_groups; ++h) {
        float* lg = slog + h * seg;
        float m = -INFINITY;
        for (int t = lane; t < seg; t += 32) m = fmaxf(m, lg[t]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float l = 0.f;
        for (int t = lane; t < seg; t += 32) {
          // a warp's share may be all -inf beside finite logits of the page's other warps: it weighs nothing
          const float pt = wpp > 1 && lg[t] == -INFINITY ? 0.f : __expf(lg[t] - m);
          lg[t] = pt;
          l += pt;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) {
          float* po = wpp > 1 ? fold + h * (dh + 2)
                              : partial_out + ((int64_t)(hq0 + h) * max_blocks + page_idx) * (dh + 2);
          po[0] = m;
          po[1] = l;
        }
      }
      __syncwarp();
      // V accumulation: a lane owns 4 dimensions, one pass over the rows feeds four heads
      for (int h0 = 0; h0 < kv_groups; h0 += 4) {
        for (int d0 = 4 * lane; d0 < dh; d0 += 128) {
          float acc[4][4];
#pragma unroll
          for (int hh = 0; hh < 4; ++hh) acc[hh][0] = acc[hh][1] = acc[hh][2] = acc[hh][3] = 0.f;
          const __half* vp = v_rows + d0;
#pragma unroll 8
          for (int t = 0; t < seg; ++t) {
            const uint2 raw = *reinterpret_cast<const uint2*>(vp + t * dh);
            const float2 va = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
            const float2 vb = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
#pragma unroll
            for (int hh = 0; hh < 4; ++hh) {
              if (h0 + hh < kv_groups) {
                const float pt = slog[(h0 + hh) * seg + t];
                acc[hh][0] += pt * va.x;
                acc[hh][1] += pt * va.y;
                acc[hh][2] += pt * vb.x;
                acc[hh][3] += pt * vb.y;
              }
            }
          }
#pragma unroll
          for (int hh = 0; hh < 4; ++hh) {
            if (h0 + hh < kv_groups) {
              float* po = (wpp > 1 ? fold + (h0 + hh) * (dh + 2)
                                   : partial_out + ((int64_t)(hq0 + h0 + hh) * max_blocks + page_idx) * (dh + 2)) + 2 + d0;
              *reinterpret_cast<float2*>(po) = make_float2(acc[hh][0], acc[hh][1]);
              *reinterpret_cast<float2*>(po + 2) = make_float2(acc[hh][2], acc[hh][3]);
            }
          }
        }
      }
    }
    __syncwarp();  // this warp is done with its staged rows
    issue_stage(phys_next);
    if (wpp > 1) {  // the page's wpp triples -> one
      __syncthreads();
      if (phys >= 0) {
        const float* f0 = fold_all + (int64_t)group * wpp * kv_groups * (dh + 2);
        const int64_t fstride = (int64_t)kv_groups * (dh + 2);
        for (int i = sub * 32 + lane; i < kv_groups * (dh + 1); i += wpp * 32) {
          const int h = i / (dh + 1), e = i - h * (dh + 1) + 1;  // 1 = the sum, 2 .. the accumulator
          const float* fh = f0 + h * (dh + 2);
          float m = fh[0];
          for (int w = 1; w < wpp; ++w) m = fmaxf(m, fh[w * fstride]);
          float x = 0.f;
          for (int w = 0; w < wpp; ++w) x += fh[w * fstride + e] * __expf(fh[w * fstride] - m);
          float* po = partial_out + ((int64_t)(hq0 + h) * max_blocks + page_idx) * (dh + 2);
          po[e] = x;
          if (e == 1) po[0] = m;
        }
      }
      __syncthreads();
    }
  }
}

// log-sum-exp merge of the page partials (decode_kernel.cu:221-246).  The reference folds the
// pages into a running (max, sum, acc) one after the other; here the maximum over the pages is
// found first and every page is weighted by exp(m_page - max) directly, which gives the same
// result without a serial chain of rescales: one CTA per query head, pages in chunks whose
// weights are shared through shared memory, threads over the head dimension.
constexpr int kReduceThreads = 1024;  // 32 dimension lanes x 32 page lanes
constexpr int kReduceChunk = 1024;

// grid (query heads, dh / 32): a CTA owns 32 output dimensions of one head
__global__ void __launch_bounds__(kReduceThreads) pool_reduce_kernel(const float* __restrict__ partial_out,
                                                                     float* __restrict__ out, int dh,
                                                                     int max_pages) {
  const int hq = blockIdx.x, tid = threadIdx.x, lane = tid & 31, pl = tid >> 5;  // lane = dimension lane
  const int d = blockIdx.y * 32 + lane;
  __shared__ float s_w[kReduceChunk];
  __shared__ float s_red[32];
  __shared__ float s_acc[32][33];
  __shared__ float s_l[32];
  griddep_wait();
  griddep_launch();
  const float* base = partial_out + (int64_t)hq * max_pages * (dh + 2);
  const int64_t row = dh + 2;
  float M = -INFINITY;
  for (int pg = tid; pg < max_pages; pg += kReduceThreads) {
    const float m_s = base[pg * row], l_s = base[pg * row + 1];
    if (!(m_s == -INFINITY && l_s == 0.f)) M = fmaxf(M, m_s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  if (lane == 0) s_red[pl] = M;
  __syncthreads();
  M = s_red[0];
  for (int i = 1; i < 32; ++i) M = fmaxf(M, s_red[i]);
  float l_f = 0.f, a_f = 0.f;
  for (int p0 = 0; p0 < max_pages; p0 += kReduceChunk) {
    const int np = min(kReduceChunk, max_pages - p0);
    __syncthreads();
    for (int i = tid; i < np; i += kReduceThreads) {
      const float m_s = base[(p0 + i) * row], l_s = base[(p0 + i) * row + 1];
      s_w[i] = (m_s == -INFINITY && l_s == 0.f) ? 0.f : __expf(m_s - M);
    }
    __syncthreads();
    // every page row was written by pool_page_kernel (zeros for holes): zero weights need no branch
#pragma unroll 4
    for (int i = pl; i < np; i += 32) {
      const float w = s_w[i];
      const float* pr = base + (p0 + i) * row;
      l_f += w * pr[1];
      if (d < dh) a_f += w * pr[2 + d];
    }
  }
  // fold the 32 page lanes in a fixed order
  s_acc[pl][lane] = a_f;
  if (lane == 0) s_l[pl] = l_f;
  __syncthreads();
  if (pl == 0 && d < dh) {
    float l_t = 0.f, a_t = 0.f;
    for (int k = 0; k < 32; ++k) {
      l_t += s_l[k];
      a_t += s_acc[k][lane];
    }
    out[(int64_t)hq * dh + d] = a_t / (l_t + 1e-8f);
  }
}

// ---- encode + append of one token per KV head, decode_kernel.cu:10-84 -----------------------
// grid = KV heads, block = 32 * G: warp = group, lanes split the centroids.  The arithmetic
// lives in pool_append_token (common.cuh), shared with the device-bookkeeping step kernel.
__global__ void pool_encode_append_kernel(
    const float* __restrict__ k_post, const float* __restrict__ v_new,
    const float* __restrict__ decode_cb, uint8_t* __restrict__ theta_codes,
    uint8_t* __restrict__ radius_codes, float* __restrict__ r_scales, __half* __restrict__ v_pool,
    const int64_t* __restrict__ pids, int slot, int G, int g, int C, int G_max, int dh,
    int page_size, int is_new_page) {
  griddep_wait();
  griddep_launch();
  pool_append_token(k_post, v_new, decode_cb, theta_codes, radius_codes, r_scales, v_pool,
                    pids[blockIdx.x], slot, G, g, C, G_max, dh, page_size, is_new_page);
}

// ---- logits from a precomputed q.centroid table (new_fused_decode.cpp:3-22) ------------------
// q_lut f32 [Hq][num_tiers][G_max][cb_size_max]; logits_out f32 [Hq][max_blocks*page_size].
// Holes, slots past ctx_lens and exact-zero logits get the -1e9 sentinel of
// decode_kernel.cu:194.  Tier geometry comes from the table itself: groups >= G of a tier
// have zero radius codes in the pool and contribute nothing.
__global__ void qlut_logits_kernel(const float* __restrict__ q_lut,
                                   const uint8_t* __restrict__ theta_codes,
                                   const uint8_t* __restrict__ radius_codes,
                                   const float* __restrict__ r_scales,
                                   const int* __restrict__ block_table,
                                   const int* __restrict__ bits_table,
                                   const int* __restrict__ ctx_lens, float* __restrict__ logits_out,
                                   int num_q_heads, int kv_groups, int num_tiers, int max_blocks,
                                   int page_size, int G_max, int cb_size_max, float sm_scale) {
  const int hkv = blockIdx.x, page_idx = blockIdx.y;
  const int phys = block_table[hkv * max_blocks + page_idx];
  const int tier_idx = phys >= 0 ? bits_table[hkv * max_blocks + page_idx] : 0;
  const int ctx = ctx_lens ? ctx_lens[hkv] : max_blocks * page_size;
  for (int i = threadIdx.x; i < kv_groups * page_size; i += blockDim.x) {
    const int h = i / page_size, t = i - h * page_size;
    const int hq = hkv * kv_groups + h;
    float outv = -1e9f;
    if (phys >= 0 && page_idx * page_size + t < ctx) {
      const uint8_t* th = theta_codes + ((int64_t)phys * page_size + t) * G_max;
      const uint8_t* rc = radius_codes + ((int64_t)phys * page_size + t) * G_max;
      const float* lut = q_lut + ((int64_t)hq * num_tiers + tier_idx) * G_max * cb_size_max;
      float s = 0.f;
      for (int gg = 0; gg < G_max; ++gg) {
        const float r_hat = r_scales[(int64_t)phys * G_max + gg] * (float)rc[gg] / 255.0f;
        s += r_hat * lut[gg * cb_size_max + th[gg]];
      }
      if (s != 0.f) outv = s * sm_scale;
    }
    logits_out[(int64_t)hq * max_blocks * page_size + (int64_t)page_idx * page_size + t] = outv;
  }
}

// ---- logits over bit-packed byte pages with per-token back-rotation --------------------------
// Restates spherical_kv_pipeline.py:2143-2176 per (token, query head): rotate q by the key
// position with the caller's HF-layout tables, normalise per group, clamp the cosine,
// weight by the de-quantised radius.  Output [Hq][n_pages * page_size]; slots with
// position < 0 or past the page count, and heads outside the page's KV head, get 0.
__global__ void ragged_logits_kernel(const uint8_t* __restrict__ pages,
                                     const int* __restrict__ ptable,
                                     const int* __restrict__ head_ids,
                                     const int* __restrict__ positions,
                                     const float* __restrict__ cos_tbl,
                                     const float* __restrict__ sin_tbl, const float* __restrict__ q,
                                     const float* __restrict__ codebooks,
                                     float* __restrict__ logits_out, int grp, int num_kv, int dh,
                                     int G, int g, int b_theta, int page_size, int n_pages, int Hq,
                                     int table_rows, int radius_fmt) {
  const int pg = blockIdx.x;
  const int hkv = head_ids[pg];
  const int poff = ptable[3 * pg], toff = ptable[3 * pg + 1], roff = ptable[3 * pg + 2];
  const int count = pages[poff + 1];
  const int C = 1 << b_theta, half = dh >> 1;
  const float inv_sqrt = rsqrtf((float)dh);
  const int64_t out_stride = (int64_t)n_pages * page_size;
  for (int i = threadIdx.x; i < Hq * page_size; i += blockDim.x) {
    const int hq = i / page_size, t = i - hq * page_size;
    float outv = 0.f;
    const int pos = positions[(int64_t)pg * page_size + t];
    if (hq / grp == hkv && hkv < num_kv && t < count && pos >= 0 && pos < table_rows) {
      const float* qh = q + (int64_t)hq * dh;
      const float* cr = cos_tbl + (int64_t)pos * dh;
      const float* sr = sin_tbl + (int64_t)pos * dh;
      for (int gg = 0; gg < G; ++gg) {
        const int64_t bit = ((int64_t)t * G + gg) * b_theta;
        uint32_t w = 0;
        for (int bb = 0; bb < 2; ++bb) w |= (uint32_t)pages[toff + (bit >> 3) + bb] << (8 * bb);
        const int code = (int)((w >> (bit & 7)) & (uint32_t)(C - 1));
        float rad;
        if (radius_fmt == SPHKV_RADIUS_F16) {
          const uint16_t hv = (uint16_t)pages[roff + 2 * (t * G + gg)] |
                              ((uint16_t)pages[roff + 2 * (t * G + gg) + 1] << 8);
          rad = __half2float(__ushort_as_half(hv));
        } else {
          float sc;
          memcpy(&sc, pages + poff + 8 + 4 * gg, 4);
          rad = sc * (float)(int8_t)pages[roff + t * G + gg] / 127.0f;
        }
        const float* cw = codebooks + ((int64_t)(hkv * G + gg) * C + code) * g;
        float nsq = 0.f, dot = 0.f;
        for (int d = 0; d < g; ++d) {
          const int dd = gg * g + d;
          const float rh = dd < half ? -qh[dd + half] : qh[dd - half];
          const float qr = qh[dd] * cr[dd] - rh * sr[dd];
          nsq += qr * qr;
          dot += qr * cw[d];
        }
        const float qn = fmaxf(sqrtf(nsq), 1e-6f);
        const float cpg = fminf(fmaxf(dot / qn, -1.f), 1.f);
        outv += qn * cpg * rad;
      }
      outv *= inv_sqrt;
    }
    logits_out[(int64_t)hq * out_stride + (int64_t)pg * page_size + t] = outv;
  }
}

// The same logits for the shapes models use (dh 64 or 128, g 16 or 32, float4-aligned tables).  The
// kernel above walks one (token, query head) per thread: every lane gathers its own cos/sin row and
// codebook row a float at a time, and the query is rotated from global memory for each group.  Here a
// token's dh dimensions lie across dh / 4 lanes, four each, so a cos, sin or centroid row is one
// coalesced 16-byte load per lane, the rotation partner of a lane's four dimensions is loaded with them,
// and four query heads live in registers over all of a warp's tokens.  Per group the (norm, dot) pairs
// of the four heads are reduced and transposed at once (three shuffles each): lane j of a quad ends with
// head j and does that head's square root and division.  A CTA covers kRagSlots slots of one page and
// also writes the zeros of the other heads.  Bound: latency at a few thousand tokens, the cos/sin rows
// from L2 beyond.  2458 tokens x 8 KV heads, 32 query heads: 167 -> 11 us.
constexpr int kRagSlots = 32, kRagWarps = 4;
template <int DH, int LG>  // LG = lanes per group = g / 4
__global__ void __launch_bounds__(kRagWarps * 32) ragged_logits_rows_kernel(
    const uint8_t* __restrict__ pages, const int* __restrict__ ptable, const int* __restrict__ head_ids,
    const int* __restrict__ positions, const float* __restrict__ cos_tbl, const float* __restrict__ sin_tbl,
    const float* __restrict__ q, const float* __restrict__ codebooks, float* __restrict__ logits_out, int grp,
    int num_kv, int b_theta, int page_size, int n_pages, int Hq, int table_rows, int radius_fmt) {
  constexpr int LPT = DH / 4, TPW = 32 / LPT;  // lanes per token, tokens a warp works on at once
  constexpr int G = LPT / LG, g = 4 * LG;
  constexpr int kPerWarp = kRagSlots / kRagWarps;      // slots of a warp
  __shared__ float s_out[4][kRagSlots];
  const int pg = blockIdx.x, slot0 = blockIdx.y * kRagSlots;
  const int n_slots = min(kRagSlots, page_size - slot0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l = lane & (LPT - 1), sub = lane / LPT, d = 4 * l, gg = l / LG, j = l & 3;
  const int hkv = head_ids[pg];
  const bool known = hkv >= 0 && hkv < num_kv;
  const int poff = ptable[3 * pg], toff = ptable[3 * pg + 1], roff = ptable[3 * pg + 2];
  const int count = pages[poff + 1];
  const int64_t out_stride = (int64_t)n_pages * page_size;
  float* out_pg = logits_out + (int64_t)pg * page_size + slot0;
  // rows of the other KV heads
  for (int i = threadIdx.x; i < Hq * kRagSlots; i += kRagWarps * 32) {
    const int hq = i / kRagSlots, t = i & (kRagSlots - 1);
    if (t < n_slots && !(known && hq / grp == hkv)) out_pg[hq * out_stride + t] = 0.f;
  }
  if (!known) return;
  float sc = 0.f;
  memcpy(&sc, pages + poff + 8 + 4 * gg, 4);
  const float* cb = codebooks + (((int64_t)hkv * G + gg) << b_theta) * g + (d & (g - 1));
  const float inv_sqrt = rsqrtf((float)DH);
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int h0 = 0; h0 < grp; h0 += 4) {
    float4 qa[4], qb[4];  // the lane's dimensions, and what rotate_half pairs them with
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const float* qh = q + ((int64_t)hkv * grp + h0 + h) * DH;
      qa[h] = h0 + h < grp ? *reinterpret_cast<const float4*>(qh + d) : zero4;
      const float4 p = h0 + h < grp ? *reinterpret_cast<const float4*>(qh + (d ^ (DH / 2))) : zero4;
      qb[h] = d < DH / 2 ? make_float4(-p.x, -p.y, -p.z, -p.w) : p;
    }
#pragma unroll 2
    for (int i = 0; i < kPerWarp; i += TPW) {
      const int ts = warp * kPerWarp + i + sub, t = slot0 + ts;
      const int pos = ts < n_slots ? positions[(int64_t)pg * page_size + t] : -1;
      const bool live = ts < n_slots && t < count && pos >= 0 && pos < table_rows;
      float4 cs = zero4, sn = zero4, cw = zero4;
      float rad = 0.f;
      if (live) {
        cs = __ldg(reinterpret_cast<const float4*>(cos_tbl + (int64_t)pos * DH + d));
        sn = __ldg(reinterpret_cast<const float4*>(sin_tbl + (int64_t)pos * DH + d));
        const int64_t bit = ((int64_t)t * G + gg) * b_theta;
        const uint32_t w = (uint32_t)pages[toff + (bit >> 3)] | ((uint32_t)pages[toff + (bit >> 3) + 1] << 8);
        const int code = (int)((w >> (bit & 7)) & ((1u << b_theta) - 1u));
        cw = __ldg(reinterpret_cast<const float4*>(cb + code * g));
        if (radius_fmt == SPHKV_RADIUS_F16) {
          const uint16_t hv = (uint16_t)pages[roff + 2 * (t * G + gg)] |
                              (uint16_t)((uint16_t)pages[roff + 2 * (t * G + gg) + 1] << 8);
          rad = __half2float(__ushort_as_half(hv));
        } else {
          rad = sc * (float)(int8_t)pages[roff + t * G + gg] / 127.0f;
        }
      }
      float nsq[4], dot[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float x0 = qa[h].x * cs.x - qb[h].x * sn.x, x1 = qa[h].y * cs.y - qb[h].y * sn.y;
        const float x2 = qa[h].z * cs.z - qb[h].z * sn.z, x3 = qa[h].w * cs.w - qb[h].w * sn.w;
        nsq[h] = (x0 * x0 + x1 * x1) + (x2 * x2 + x3 * x3);
        dot[h] = (x0 * cw.x + x1 * cw.y) + (x2 * cw.z + x3 * cw.w);
      }
      auto fold = [&](const float (&v)[4]) -> float {  // sum over the group's lanes; lane j keeps head j
        const bool odd = j & 1, up = j & 2;
        const float k0 = (odd ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], 1);
        const float k1 = (odd ? v[3] : v[2]) + __shfl_xor_sync(0xffffffffu, odd ? v[2] : v[3], 1);
        float r = (up ? k1 : k0) + __shfl_xor_sync(0xffffffffu, up ? k0 : k1, 2);
        if (LG == 8) r += __shfl_xor_sync(0xffffffffu, r, 4);
        return r;
      };
      const float qn = fmaxf(sqrtf(fold(nsq)), 1e-6f);
      const float cpg = fminf(fmaxf(fold(dot) / qn, -1.f), 1.f);
      float logit = qn * cpg * rad;
#pragma unroll
      for (int o = LG; o < LPT; o <<= 1) logit += __shfl_xor_sync(0xffffffffu, logit, o);
      if (l < 4) s_out[j][ts] = live ? logit * inv_sqrt : 0.f;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * kRagSlots; i += kRagWarps * 32) {
      const int h = i / kRagSlots, t = i & (kRagSlots - 1);
      if (h0 + h < grp && t < n_slots) out_pg[((int64_t)hkv * grp + h0 + h) * out_stride + t] = s_out[h][t];
    }
    __syncthreads();
  }
}

}  // namespace sphkv

using namespace sphkv;

static int sphkv_sm_count_or(int fallback) {
  const int sms = sm_count_current_device();
  return sms > 0 ? sms : fallback;
}

extern "C" int sphkv_pool_decode(const float* q_all, const float* cb_flat, const int32_t* tier_G,
                                 const int32_t* tier_g, const uint8_t* theta_codes,
                                 const uint8_t* radius_codes, const float* r_scales,
                                 const void* v_pool, const int32_t* block_table,
                                 const int32_t* bits_table, const int32_t* ctx_lens, float* out,
                                 float* partial_scratch, int32_t num_q_heads, int32_t num_kv_heads,
                                 int32_t kv_groups, int32_t num_tiers, int32_t max_blocks,
                                 int32_t page_size, int32_t dh, int32_t G_max, int32_t cb_max,
                                 int32_t g_max, float sm_scale, int32_t max_ctx, void* stream) {
  (void)ctx_lens;  // validity is encoded by block_table == -1 and the zero-logit sentinel,
  (void)max_ctx;   // as in decode_kernel.cu:120,139-144,194
  SPHKV_REQUIRE(q_all && cb_flat && tier_G && tier_g && theta_codes && radius_codes && r_scales &&
                    v_pool && block_table && bits_table && out && partial_scratch,
                SPHKV_E_ARG, "pool_decode: NULL pointer");
  SPHKV_REQUIRE(num_q_heads > 0 && num_kv_heads > 0 && kv_groups > 0 &&
                    num_q_heads == num_kv_heads * kv_groups,
                SPHKV_E_ARG, "pool_decode: Hq=%d Hkv=%d groups=%d", num_q_heads, num_kv_heads,
                kv_groups);
  SPHKV_REQUIRE(max_blocks > 0 && page_size > 0 && dh > 0 && dh <= 512 && (dh & 3) == 0 && G_max > 0 &&
                    cb_max > 0 && g_max > 0 && num_tiers > 0,
                SPHKV_E_ARG, "pool_decode: bad size");
  SPHKV_REQUIRE((reinterpret_cast<uintptr_t>(v_pool) & 7) == 0 && (reinterpret_cast<uintptr_t>(partial_scratch) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(theta_codes) & 3) == 0 && (reinterpret_cast<uintptr_t>(radius_codes) & 3) == 0,
                SPHKV_E_ALIGN, "pool_decode: v_pool / partial_scratch need 8 B, code arrays 4 B alignment");
  auto smem_for = [&](int wpp) -> size_t {
    return ((size_t)kv_groups * dh + (((size_t)num_tiers * kv_groups * G_max * cb_max + 1) & ~(size_t)1) +
            (size_t)kPoolWarps * ((size_t)kv_groups * (page_size / wpp) + G_max) +
            (wpp > 1 ? (size_t)kPoolWarps * kv_groups * (dh + 2) : 0)) * sizeof(float);
  };
  // warps that share a page: as many as leave each 16 tokens (and fit shared memory)
  int wpp = kPoolWarps;
  while (wpp > 1 && (page_size % wpp != 0 || page_size / wpp < 16 || smem_for(wpp) > 100 * 1024)) wpp >>= 1;
  size_t smem = smem_for(wpp);
  SPHKV_REQUIRE(smem <= 200 * 1024, SPHKV_E_LIMIT, "pool_decode: needs %zu B shared memory", smem);
  // asynchronous staging of a warp's rows: 16-byte pieces, and two CTAs per SM have to stay possible
  const int seg = page_size / wpp;
  int stage_bytes = seg * dh * 2 + 2 * seg * G_max;
  if (((seg * G_max) & 15) != 0 || (dh & 7) != 0 || smem + 16 + (size_t)kPoolWarps * stage_bytes > 110 * 1024 ||
      ((reinterpret_cast<uintptr_t>(v_pool) | reinterpret_cast<uintptr_t>(theta_codes) |
        reinterpret_cast<uintptr_t>(radius_codes)) & 15) != 0)
    stage_bytes = 0;
  if (stage_bytes > 0) smem = (smem + 15) / 16 * 16 + (size_t)kPoolWarps * stage_bytes;
  {
    static SmemOptIn opt_in;
    if (int rc = ensure_dynamic_smem(opt_in, (const void*)pool_page_kernel, (int)smem, "pool_decode")) return rc;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // rounds of pages per CTA: up to kMaxPageRounds (amortises the table build), fewer while the grid is small
  const int at_once = kPoolWarps / wpp;
  int rounds = (int)(((int64_t)num_kv_heads * max_blocks) / ((int64_t)at_once * 2 * sphkv_sm_count_or(148)));
  rounds = rounds < 1 ? 1 : (rounds > kMaxPageRounds ? kMaxPageRounds : rounds);
  rounds = std::max(rounds, (int)((max_blocks + (int64_t)at_once * 65535 - 1) / ((int64_t)at_once * 65535)));  // grid.y
  const int ppc = at_once * rounds;
  (void)launch_overlapped(pool_page_kernel, dim3(num_kv_heads, (max_blocks + ppc - 1) / ppc), dim3(kPoolThreads), smem, st,
      q_all, cb_flat, tier_G, tier_g, theta_codes, radius_codes, r_scales,
      reinterpret_cast<const __half*>(v_pool), block_table, bits_table, partial_scratch,
      num_q_heads, kv_groups, num_tiers, max_blocks, page_size, dh, G_max, cb_max, g_max, sm_scale, wpp, rounds,
      stage_bytes);
  if (int rc = check_launch("pool_page_kernel")) return rc;
  (void)launch_overlapped(pool_reduce_kernel, dim3(num_q_heads, (dh + 31) / 32), dim3(kReduceThreads), 0, st,
                          static_cast<const float*>(partial_scratch), out, dh, max_blocks);
  return check_launch("pool_reduce_kernel");
}

extern "C" int sphkv_pool_encode_append(const float* k_post, const float* v_new,
                                        const float* decode_cb, uint8_t* theta_codes,
                                        uint8_t* radius_codes, float* r_scales, void* v_pool,
                                        const int64_t* pids, int32_t slot, int32_t G, int32_t g,
                                        int32_t C, int32_t G_max, int32_t dh, int32_t page_size,
                                        int32_t is_new_page, int32_t num_kv, void* stream) {
  SPHKV_REQUIRE(k_post && v_new && decode_cb && theta_codes && radius_codes && r_scales && v_pool &&
                    pids,
                SPHKV_E_ARG, "encode_append: NULL pointer");
  SPHKV_REQUIRE(num_kv > 0 && G > 0 && G <= 32 && g > 0 && C > 0 && G <= G_max && G * g <= dh &&
                    slot >= 0 && slot < page_size,
                SPHKV_E_ARG, "encode_append: G=%d g=%d C=%d G_max=%d dh=%d slot=%d page_size=%d", G,
                g, C, G_max, dh, slot, page_size);
  (void)launch_overlapped(pool_encode_append_kernel, dim3(num_kv), dim3(32 * G), 0, reinterpret_cast<cudaStream_t>(stream),
      k_post, v_new, decode_cb, theta_codes, radius_codes, r_scales,
      reinterpret_cast<__half*>(v_pool), pids, slot, G, g, C, G_max, dh, page_size, is_new_page);
  return check_launch("pool_encode_append_kernel");
}

extern "C" int sphkv_qlut_logits(const float* q_lut, const uint8_t* theta_codes,
                                 const uint8_t* radius_codes, const float* r_scales,
                                 const int32_t* block_table, const int32_t* bits_table,
                                 const int32_t* ctx_lens, float* logits_out, int32_t num_q_heads,
                                 int32_t num_kv_heads, int32_t kv_groups, int32_t num_tiers,
                                 int32_t max_blocks, int32_t page_size, int32_t G_max,
                                 int32_t cb_size_max, float sm_scale, int32_t max_ctx,
                                 void* stream) {
  (void)max_ctx;
  SPHKV_REQUIRE(q_lut && theta_codes && radius_codes && r_scales && block_table && bits_table &&
                    logits_out,
                SPHKV_E_ARG, "qlut_logits: NULL pointer");
  SPHKV_REQUIRE(num_q_heads > 0 && num_kv_heads > 0 && num_q_heads == num_kv_heads * kv_groups &&
                    max_blocks > 0 && page_size > 0 && G_max > 0 && cb_size_max > 0 && num_tiers > 0,
                SPHKV_E_ARG, "qlut_logits: bad size");
  qlut_logits_kernel<<<dim3(num_kv_heads, max_blocks), 128, 0,
                       reinterpret_cast<cudaStream_t>(stream)>>>(
      q_lut, theta_codes, radius_codes, r_scales, block_table, bits_table, ctx_lens, logits_out,
      num_q_heads, kv_groups, num_tiers, max_blocks, page_size, G_max, cb_size_max, sm_scale);
  return check_launch("qlut_logits_kernel");
}

extern "C" int sphkv_ragged_logits(const uint8_t* pages, const int32_t* ptable,
                                   const int32_t* head_ids, const int32_t* positions,
                                   const float* cos_tbl, const float* sin_tbl, const float* q,
                                   const float* codebooks, float* logits_out, int32_t grp,
                                   int32_t num_kv, int32_t dh, int32_t G, int32_t g, int32_t b_theta,
                                   int32_t page_size, int32_t n_pages, int32_t Hq,
                                   int32_t table_rows, int32_t radius_fmt, int32_t reserved,
                                   void* stream) {
  (void)reserved;
  SPHKV_REQUIRE(pages && ptable && head_ids && positions && cos_tbl && sin_tbl && q && codebooks &&
                    logits_out,
                SPHKV_E_ARG, "ragged_logits: NULL pointer");
  SPHKV_REQUIRE(n_pages > 0 && grp > 0 && num_kv > 0 && Hq == grp * num_kv && G * g == dh &&
                    (dh & 1) == 0 && b_theta >= 1 && b_theta <= 8 && page_size > 0 && table_rows > 0,
                SPHKV_E_ARG, "ragged_logits: bad size (Hq=%d grp=%d num_kv=%d G=%d g=%d dh=%d)", Hq,
                grp, num_kv, G, g, dh);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // one coalesced row per token where the rows are float4s across a power-of-two of lanes
  const bool rows = (dh == 64 || dh == 128) && (g == 16 || g == 32) &&
                    ((reinterpret_cast<uintptr_t>(cos_tbl) | reinterpret_cast<uintptr_t>(sin_tbl) |
                      reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(codebooks)) & 15) == 0;
  if (rows) {
    const dim3 grid(n_pages, (page_size + kRagSlots - 1) / kRagSlots);
    auto kern = dh == 128 ? (g == 16 ? ragged_logits_rows_kernel<128, 4> : ragged_logits_rows_kernel<128, 8>)
                          : (g == 16 ? ragged_logits_rows_kernel<64, 4> : ragged_logits_rows_kernel<64, 8>);
    kern<<<grid, kRagWarps * 32, 0, st>>>(pages, ptable, head_ids, positions, cos_tbl, sin_tbl, q, codebooks, logits_out, grp,
                               num_kv, b_theta, page_size, n_pages, Hq, table_rows, radius_fmt);
    return check_launch("ragged_logits_rows_kernel");
  }
  ragged_logits_kernel<<<n_pages, 256, 0, st>>>(
      pages, ptable, head_ids, positions, cos_tbl, sin_tbl, q, codebooks, logits_out, grp, num_kv,
      dh, G, g, b_theta, page_size, n_pages, Hq, table_rows, radius_fmt);
  return check_launch("ragged_logits_kernel");
}

// ---- page-level importance EMA from per-block (m, l) --------------------------------------------
// _omega_ema_eager (spherical_kv_pipeline.py:952-987) in one launch: per query head the block
// weights exp(max(m - m_max, -60)) * l are normalised over the blocks, averaged over the query
// heads of a KV head and blended into omega with factor beta.  ml points at the (m, l) pairs of
// (query head, block): element (hq, blk) lives at ml[(hq * max_blocks + blk) * stride + {0, 1}]
// (stride = dh + 2 for the partial_scratch of sphkv_pool_decode, 2 for page_ml of
// sphkv_decode_paged).  omega [n_units][max_blocks] is updated in place; unit u owns query heads
// u * kv_groups .. (u + 1) * kv_groups - 1.
namespace sphkv {
__global__ void omega_ema_kernel(const float* __restrict__ ml, float* __restrict__ omega,
                                 int kv_groups, int max_blocks, int stride, float beta) {
  const int u = blockIdx.x;
  __shared__ float s_red[32];
  __shared__ float s_val;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto block_reduce = [&](float v, bool is_max) -> float {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float t = __shfl_xor_sync(0xffffffffu, v, o);
      v = is_max ? fmaxf(v, t) : v + t;
    }
    if (lane == 0) s_red[warp] = v;
    __syncthreads();
    if (warp == 0) {
      float x = lane < nw ? s_red[lane] : (is_max ? -INFINITY : 0.f);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float t = __shfl_xor_sync(0xffffffffu, x, o);
        x = is_max ? fmaxf(x, t) : x + t;
      }
      if (lane == 0) s_val = x;
    }
    __syncthreads();
    const float r = s_val;
    __syncthreads();
    return r;
  };
  // mass accumulated over the group's query heads, blocks strided over the threads
  extern __shared__ float s_mass[];  // [max_blocks]
  for (int i = threadIdx.x; i < max_blocks; i += blockDim.x) s_mass[i] = 0.f;
  __syncthreads();
  for (int h = 0; h < kv_groups; ++h) {
    const float* base = ml + ((int64_t)(u * kv_groups + h) * max_blocks) * stride;
    float mx = -1e30f;
    for (int i = threadIdx.x; i < max_blocks; i += blockDim.x) {
      const float m = base[(int64_t)i * stride], l = base[(int64_t)i * stride + 1];
      mx = fmaxf(mx, l > 0.f ? m : -1e30f);
    }
    mx = block_reduce(mx, true);
    float z = 0.f;
    for (int i = threadIdx.x; i < max_blocks; i += blockDim.x) {
      const float m = base[(int64_t)i * stride], l = base[(int64_t)i * stride + 1];
      const float ms = l > 0.f ? m : -1e30f;
      z += __expf(fmaxf(ms - mx, -60.f)) * l;
    }
    z = fmaxf(block_reduce(z, false), 1e-12f);
    for (int i = threadIdx.x; i < max_blocks; i += blockDim.x) {
      const float m = base[(int64_t)i * stride], l = base[(int64_t)i * stride + 1];
      const float ms = l > 0.f ? m : -1e30f;
      s_mass[i] += __expf(fmaxf(ms - mx, -60.f)) * l / z;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < max_blocks; i += blockDim.x) {
    float* o = omega + (int64_t)u * max_blocks + i;
    *o = *o * beta + (s_mass[i] / (float)kv_groups) * (1.0f - beta);
  }
}
}  // namespace sphkv

extern "C" int sphkv_omega_ema(const float* ml, float* omega, int32_t n_units, int32_t kv_groups,
                               int32_t max_blocks, int32_t stride, float beta, void* stream) {
  SPHKV_REQUIRE(ml && omega, SPHKV_E_ARG, "omega_ema: NULL pointer");
  SPHKV_REQUIRE(n_units > 0 && kv_groups > 0 && max_blocks > 0 && stride >= 2, SPHKV_E_ARG,
                "omega_ema: n_units=%d kv_groups=%d max_blocks=%d stride=%d", n_units, kv_groups,
                max_blocks, stride);
  SPHKV_REQUIRE((size_t)max_blocks * 4 <= 160 * 1024, SPHKV_E_LIMIT,
                "omega_ema: max_blocks=%d exceeds 40960", max_blocks);
  const size_t smem = (size_t)max_blocks * 4;
  {
    static sphkv::SmemOptIn opt_in;
    if (int rc = sphkv::ensure_dynamic_smem(opt_in, (const void*)sphkv::omega_ema_kernel, (int)smem, "omega_ema"))
      return rc;
  }
  sphkv::omega_ema_kernel<<<n_units, 256, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      ml, omega, kv_groups, max_blocks, stride, beta);
  return sphkv::check_launch("omega_ema_kernel");
}
