// Spherical encode + page build.
//
// One CTA encodes bundles of 128 token slots (128/page_size pages) that share a (KV head,
// tier slot): warp = group, lane = four tokens (every centroid row read from shared memory
// feeds four dot products).  Per
// (token, group) the kernel computes the group radius and the nearest centroid, then the
// CTA assembles each page image in shared memory in the reference byte layout
//   [tier_id u8][count u8][fmt u8][5 x 0][G x f32 scale][LSB-first packed theta][radii]
// (paging.py:20-31, pagebuilder.py:8-33, bitpacking.py:5-29) and copies it out, together
// with the dense 16-bit V page.
//
// Arithmetic order (what "bit-exact" is defined against):
//   nsq   = fma chain d = 0..g-1 of k_d * k_d starting from 0;  r = sqrt(nsq)   (IEEE)
//   sim_c = fma chain d = 0..g-1 of k_d * cb[c][d] starting from 0
//   theta = first c maximising sim_c (strict >), as torch.argmax / decode_kernel.cu:45-55
//   scale = max_t r ; code = clamp(rint((r / max(scale, 1e-8)) * 127), -127, 127)
// The similarity is taken on the un-normalised group vector: dividing by r first
// (spherical_kv_pipeline.py:1138) scales every sim_c by the same positive factor.
#include <algorithm>

#include "search.cuh"

namespace sphkv {

struct EncodeArgs {
  sphkv_encode_params p;
  int bundles_per_cta;
  int page_smem_bytes;  // page assembly: shared memory of one page
  int wpp_shift;        // page assembly: log2 of the warps of a page
  int search_kbuf;      // search launch: byte offset of the staged rows
  int search_chunk;     // search launch: consecutive bundles a CTA takes at a time (1 .. 8)
};

constexpr int kEncThreads = 256;

// two 16-bit elements (bf16 or f16) of one 32-bit word, widened exactly
__device__ __forceinline__ void unpack16(uint32_t w, int dtype, float& lo, float& hi) {
  if (dtype == SPHKV_BF16) {
    lo = __uint_as_float(w << 16);
    hi = __uint_as_float(w & 0xFFFF0000u);
  } else {
    const __half2 h = *reinterpret_cast<const __half2*>(&w);
    lo = __low2float(h);
    hi = __high2float(h);
  }
}

template <int GS>
__device__ __forceinline__ void load_group(const void* base, int dtype, int64_t off, float (&k)[GS]) {
  if (dtype == SPHKV_F32 && (((uintptr_t)base + off * 4) & 15) == 0) {
    const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + off);
#pragma unroll
    for (int i = 0; i < GS / 4; ++i) {
      const float4 v = ldg_stream_f4(s + i);
      k[4 * i] = v.x; k[4 * i + 1] = v.y; k[4 * i + 2] = v.z; k[4 * i + 3] = v.w;
    }
  } else if (dtype != SPHKV_F32 && (((uintptr_t)base + off * 2) & 15) == 0) {
    const uint4* s =
        reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + off);
#pragma unroll
    for (int i = 0; i < GS / 8; ++i) {
      const uint4 v = __ldg(s + i);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) unpack16(w[e], dtype, k[8 * i + 2 * e], k[8 * i + 2 * e + 1]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < GS; ++i) k[i] = load_as_float(base, dtype, off + i);
  }
}

// Eight consecutive V elements starting at element offset `off` of v_src, as one 16-byte chunk
// of the 16-bit V pool (copied when the types agree, else rounded to nearest even).
__device__ __forceinline__ uint4 load_v_chunk(const sphkv_encode_params& p, bool same, int64_t off) {
  if (same && (((uintptr_t)p.v_src + off * 2) & 15) == 0)
    return __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.v_src) + off));
  float v[8];
  if (p.v_src_dtype == SPHKV_F32 && (((uintptr_t)p.v_src + off * 4) & 15) == 0) {
    const float4 a0 = ldg_stream_f4(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.v_src) + off));
    const float4 a1 = ldg_stream_f4(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.v_src) + off + 4));
    v[0] = a0.x; v[1] = a0.y; v[2] = a0.z; v[3] = a0.w;
    v[4] = a1.x; v[5] = a1.y; v[6] = a1.z; v[7] = a1.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = load_as_float(p.v_src, p.v_src_dtype, off + e);
  }
  uint32_t w[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (p.v_pool_dtype == SPHKV_F16) {
      w[e] = pack_f16x2(v[2 * e], v[2 * e + 1]);
    } else {
      __nv_bfloat162 hb2 = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
      w[e] = *reinterpret_cast<uint32_t*>(&hb2);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

constexpr int kMaxBundlesPerCta = 8;  // consecutive bundles one CTA walks (they mostly share a codebook)

// Squared norm and nearest centroid of TOK tokens' GS-dim group vectors: the fixed fma chains that
// define the encoder bit for bit (d = 0 .. GS-1 from 0; first maximum wins).  Every centroid row
// read from shared memory (`cbg`, [C][GS]) feeds TOK dot products.
template <int GS, int TOK>
__device__ __forceinline__ void search_tokens(const float (&k)[TOK][GS], const float* __restrict__ cbg, int C, float (&nsq)[TOK],
                                              int (&code)[TOK]) {
#pragma unroll
  for (int h = 0; h < TOK; ++h) nsq[h] = 0.f;
#pragma unroll
  for (int d = 0; d < GS; ++d)
#pragma unroll
    for (int h = 0; h < TOK; ++h) nsq[h] = __fmaf_rn(k[h][d], k[h][d], nsq[h]);
  float best[TOK];
#pragma unroll
  for (int h = 0; h < TOK; ++h) { best[h] = -INFINITY; code[h] = 0; }
  SPHKV_UNROLL_SEARCH
  for (int c = 0; c < C; ++c) {
    const float4* row = reinterpret_cast<const float4*>(cbg + c * GS);
    float sacc[TOK];
#pragma unroll
    for (int h = 0; h < TOK; ++h) sacc[h] = 0.f;
#pragma unroll
    for (int i = 0; i < GS / 4; ++i) {
      const float4 v = row[i];
#pragma unroll
      for (int h = 0; h < TOK; ++h) {
        sacc[h] = __fmaf_rn(k[h][4 * i], v.x, sacc[h]);
        sacc[h] = __fmaf_rn(k[h][4 * i + 1], v.y, sacc[h]);
        sacc[h] = __fmaf_rn(k[h][4 * i + 2], v.z, sacc[h]);
        sacc[h] = __fmaf_rn(k[h][4 * i + 3], v.w, sacc[h]);
      }
    }
#pragma unroll
    for (int h = 0; h < TOK; ++h)
      if (sacc[h] > best[h]) { best[h] = sacc[h]; code[h] = c; }
  }
}

// The codebook of one (KV head, tier slot), [G][C][GS] packed, global -> shared memory: every 16-byte copy of
// the CTA in flight at once.  The caller's barrier publishes it.
template <int GS>
__device__ __forceinline__ void stage_slot_codebook(const sphkv_encode_params& p, int head, int slot, float* cb_s) {
  const int bits = p.tiers.bits[slot], G = p.dh / GS;
  const float* src = p.codebooks + ((int64_t)(head * p.tiers.n_slots + slot) * p.tiers.G_max) * p.tiers.C_max * p.tiers.g_max;
  const uint32_t dst = smem_u32(cb_s);
  constexpr int Q4 = GS / 4;
  const int total = (G << bits) * Q4;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int q4 = i % Q4, row = i / Q4;
    const int c = row & ((1 << bits) - 1), gam = row >> bits;
    cp_async_16(dst + i * 16, src + (gam * p.tiers.C_max + c) * p.tiers.g_max + 4 * q4);
  }
  cp_async_commit();
  cp_async_wait<0>();
}

// Everything in one kernel (the route without scratch): search, page images and V pages per bundle.
// With scratch the work is split instead: search_bundles_kernel writes radius + centroid index per
// (page slot, group) and assemble_pages_kernel builds the pages, so the FMA-bound search runs without
// the barriers and small dependent loads of the page bookkeeping.
template <int GS>
__global__ void __launch_bounds__(kEncThreads) encode_bundle_kernel(const EncodeArgs a) {
  const sphkv_encode_params& p = a.p;
  extern __shared__ __align__(16) uint8_t smem[];
  const int N = p.page_size, dh = p.dh;
  constexpr int TB = 128;                   // token slots per bundle
  const int ppb = TB / N;                   // pages per bundle (page_size <= 128)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = dh / GS, g_shift = 31 - __clz(G);
  const int n_shift = 31 - __clz(N);  // page_size is a power of two
  const int rb = p.radius_fmt == SPHKV_RADIUS_F16 ? 2 : 1;
  const int C_cap = p.tiers.C_max;

  float* cb_s = reinterpret_cast<float*>(smem);                       // [G][C][GS]
  float* r_s = cb_s + G * C_cap * GS;                                  // [TB][G]
  float* scale_s = r_s + TB * G;                                       // [8][8]
  int* count_s = reinterpret_cast<int*>(scale_s + 64);                 // [8]
  int* page_s = count_s + 8;                                           // [8]
  int* poff_s = page_s + 8;                                            // [8] byte offset of each page
  uint8_t* th_s = reinterpret_cast<uint8_t*>(poff_s + 8);              // [TB][G]
  uint8_t* img = th_s + TB * G;                                        // page images, 16-aligned
  img = reinterpret_cast<uint8_t*>(((uintptr_t)img + 15) & ~(uintptr_t)15);

  int loaded_key = -1;
  const int b_first = blockIdx.x * a.bundles_per_cta;
  const int b_last = min(p.n_bundles, b_first + a.bundles_per_cta);
  for (int bi = b_first; bi < b_last; ++bi) {
    const int32_t* bundle = p.bundles + 8 * (int64_t)bi;
    __syncthreads();  // previous bundle is done with shared memory
    // ---- pages of the bundle and their valid-token counts (valid slots form a prefix) ------
    {  // 8 warps, up to 8 pages
      int page = -1, cnt = 0;
      if (warp < ppb) page = bundle[warp];
      if (page >= 0) {
        const int32_t* si = p.src_index + (int64_t)page * N;
        for (int t0 = 0; t0 < N; t0 += 32) {
          const bool ok = (t0 + lane < N) && si[t0 + lane] >= 0;
          cnt += __popc(__ballot_sync(0xffffffffu, ok));
        }
      }
      if (lane == 0) {
        count_s[warp] = cnt;
        page_s[warp] = page;
        poff_s[warp] = page >= 0 ? p.ptable[3 * (int64_t)page] : 0;
      }
    }
    __syncthreads();
    int first = -1;
    for (int q = 0; q < ppb; ++q)
      if (first < 0 && page_s[q] >= 0) first = page_s[q];
    if (first < 0) continue;
    const int head = p.page_head[first], slot = p.page_slot[first];
    if (p.tiers.g[slot] != GS) continue;  // the launch for the other group size takes this bundle
    const int bits = p.tiers.bits[slot], C = 1 << bits;
    const int img_stride = ((8 + 4 * G + (N * G * bits + 7) / 8 + N * G * rb) + 15) & ~15;

    // ---- codebook of (head, slot) -> shared memory, 128-bit copies ---------------------------
    if (head * p.tiers.n_slots + slot != loaded_key) {
      stage_slot_codebook<GS>(p, head, slot, cb_s);
      loaded_key = head * p.tiers.n_slots + slot;
      __syncthreads();
    }

    // ---- radius + nearest centroid: warp = group, lane = token slots lane + 32 h, h < 4 ----
    if (warp < G) {
      const float* cbg = cb_s + (warp << bits) * GS;
      float k[4][GS];
      bool have[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int ts = lane + 32 * h;  // token slot in bundle
        const int q = ts >> n_shift, tin = ts & (N - 1);
        const int page = page_s[q];
        int64_t row = -1;
        if (page >= 0) row = p.src_index[(int64_t)page * N + tin];
        have[h] = row >= 0;
        if (have[h]) {
          load_group<GS>(p.k_src, p.k_dtype,
                         row * p.k_row_stride + (int64_t)head * p.k_head_stride + warp * GS, k[h]);
        } else {
#pragma unroll
          for (int i = 0; i < GS; ++i) k[h][i] = 0.f;
        }
      }
      float nsq[4];
      int code[4];
      search_tokens<GS>(k, cbg, C, nsq, code);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int ts = lane + 32 * h;
        const float rv = have[h] ? __fsqrt_rn(nsq[h]) : 0.f;
        r_s[ts * G + warp] = rv;
        th_s[ts * G + warp] = (uint8_t)code[h];
      }
    }
    __syncthreads();

    // ---- per-page, per-group scale = max radius over the page's tokens ----------------------
    if (warp < ppb) {
      const int cnt = count_s[warp];
      const int tbase = warp * N;
      const int gq = lane & 7, tq = lane >> 3;
      float mx = 0.f;
      if (gq < G)
        for (int t = tq; t < cnt; t += 4) mx = fmaxf(mx, r_s[(tbase + t) * G + gq]);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
      if (lane < 8) scale_s[warp * 8 + lane] = mx;
    }
    __syncthreads();

    // ---- page images: header, scales, packed theta words ---------------------------------------
    // Every loop below runs over the whole bundle (all pages at once), so the CTA's threads share
    // the work of the 128 / page_size pages evenly instead of a fraction of them looping per page.
    const int hdr = 8 + 4 * G;
    if ((int)threadIdx.x < 2 * ppb) {
      const int q = threadIdx.x >> 1, cnt = count_s[q];
      if (cnt > 0) {
        uint32_t w = 0;
        if ((threadIdx.x & 1) == 0)
          w = (uint32_t)(p.tiers.tier_id[slot] & 0xFF) | ((uint32_t)(cnt & 0xFF) << 8) |
              ((uint32_t)(p.radius_fmt & 0xFF) << 16);
        reinterpret_cast<uint32_t*>(img + q * img_stride)[threadIdx.x & 1] = w;
      }
    }
    if ((int)threadIdx.x < 8 * ppb) {
      const int q = threadIdx.x >> 3, gq = threadIdx.x & 7;
      if (gq < G && count_s[q] > 0)
        reinterpret_cast<float*>(img + q * img_stride + 8)[gq] = scale_s[q * 8 + gq];
    }
    {
      const int max_words = ((((N * G * bits + 7) >> 3) + 3) >> 2);
      for (int it = threadIdx.x; it < ppb * max_words; it += blockDim.x) {
        const int q = it / max_words, w = it - q * max_words;
        const int nvals = count_s[q] * G;
        const int th_words = ((((nvals * bits + 7) >> 3) + 3) >> 2);
        if (w >= th_words) continue;
        const int bit0 = w * 32;
        int i = bit0 / bits;  // first value overlapping this word
        uint32_t acc = 0;
        for (; i < nvals && i * bits < bit0 + 32; ++i) {
          const uint32_t v = th_s[q * N * G + i];
          const int sh = i * bits - bit0;
          acc |= sh >= 0 ? (v << sh) : (v >> (-sh));
        }
        reinterpret_cast<uint32_t*>(img + q * img_stride + hdr)[w] = acc;
      }
    }
    __syncthreads();
    // ---- radii (may overlay the zero tail of the last theta word) ----------------------------
    for (int i = threadIdx.x; i < TB * G; i += blockDim.x) {
      const int ts = i >> g_shift, gq = i & (G - 1);
      const int q = ts >> n_shift, tin = ts & (N - 1);
      const int cnt = count_s[q];
      if (tin >= cnt) continue;
      const float rr = r_s[i];
      if (rb == 1) {
        const float safe = fmaxf(scale_s[q * 8 + gq], 1e-8f);
        float qv = rintf(__fmul_rn(__fdiv_rn(rr, safe), 127.0f));
        qv = fminf(fmaxf(qv, -127.f), 127.f);
        img[q * img_stride + hdr + ((cnt * G * bits + 7) >> 3) + tin * G + gq] = (uint8_t)(int8_t)(int)qv;
      } else {
        // stage the half's bit pattern as a 32-bit word over the radius slot (same thread
        // read it above); the bytes are laid into the page image after the barrier
        unsigned short hv;
        asm volatile("cvt.rn.f16.f32 %0, %1;" : "=h"(hv) : "f"(rr));
        reinterpret_cast<uint32_t*>(r_s)[i] = (uint32_t)hv;
      }
    }
    if (rb == 2) {
      __syncthreads();
      const uint8_t* hb = reinterpret_cast<const uint8_t*>(r_s);
      for (int b2 = threadIdx.x; b2 < 2 * TB * G; b2 += blockDim.x) {
        const int i = b2 >> 1;
        const int ts = i >> g_shift, gq = i & (G - 1);
        const int q = ts >> n_shift, tin = ts & (N - 1);
        const int cnt = count_s[q];
        if (tin >= cnt) continue;
        img[q * img_stride + hdr + ((cnt * G * bits + 7) >> 3) + 2 * (tin * G + gq) + (b2 & 1)] = hb[i * 4 + (b2 & 1)];
      }
    }
    __syncthreads();
    // ---- copy page images out -------------------------------------------------------------------
    {
      const int max_img_words = img_stride >> 2;
      for (int it = threadIdx.x; it < ppb * max_img_words; it += blockDim.x) {
        const int q = it / max_img_words, w = it - q * max_img_words;
        const int cnt = count_s[q];
        if (cnt == 0) continue;
        const int bytes = hdr + ((cnt * G * bits + 7) >> 3) + cnt * G * rb;
        if (w < (bytes >> 2))
          reinterpret_cast<uint32_t*>(p.k_pages + poff_s[q])[w] =
              reinterpret_cast<const uint32_t*>(img + q * img_stride)[w];
      }
      if ((int)threadIdx.x < 4 * ppb) {
        const int q = threadIdx.x >> 2, t = threadIdx.x & 3;
        const int cnt = count_s[q];
        if (cnt > 0) {
          const int bytes = hdr + ((cnt * G * bits + 7) >> 3) + cnt * G * rb;
          if (t < (bytes & 3)) p.k_pages[poff_s[q] + (bytes & ~3) + t] = img[q * img_stride + (bytes & ~3) + t];
        }
      }
    }

    // ---- dense V pages (16-bit), empty slots zero-filled ----------------------------------------
    // One item = 8 elements (a 16-byte output chunk) of one token slot of the bundle.  A thread
    // takes four items per round: all row lookups first, then all loads, then all stores, so four
    // independent load chains are in flight instead of one.
    if (p.v_src != nullptr && p.v_pool != nullptr) {
      constexpr int kInFlight = 4;
      const int pr_shift = 31 - __clz(dh >> 3);  // 16-byte chunks per row (dh / 8, a power of two)
      const int items = TB << pr_shift;
      const bool same = p.v_src_dtype == p.v_pool_dtype;
      for (int i0 = threadIdx.x; i0 < items; i0 += kEncThreads * kInFlight) {
        int64_t off[kInFlight], dst[kInFlight];
        bool live[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          const int i = i0 + u * kEncThreads;
          const int ts = i >> pr_shift, d = (i & ((1 << pr_shift) - 1)) * 8;
          const int page = i < items ? page_s[ts >> n_shift] : -1;
          const int tin = ts & (N - 1);
          dst[u] = -1;
          off[u] = -1;
          if (page >= 0) {
            dst[u] = (((int64_t)page * N + tin) * dh + d) >> 3;
            const int64_t row = p.src_index[(int64_t)page * N + tin];
            if (row >= 0) off[u] = row * p.v_row_stride + (int64_t)head * p.v_head_stride + d;
          }
          live[u] = off[u] >= 0;
        }
        uint4 o[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          o[u] = live[u] ? load_v_chunk(p, same, off[u]) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < kInFlight; ++u)
          if (dst[u] >= 0) reinterpret_cast<uint4*>(p.v_pool)[dst[u]] = o[u];
      }
    }
  }
}

// ---- search only (the split route) ---------------------------------------------------------
// Radius and nearest centroid of every token slot of every bundle, written to the scratch arrays
// r[(page * N + slot) * (dh / 16) + group] (f32) and theta[...] (u8).  Persistent: CTA c of n takes
// the chunks c, c + n, c + 2n, ... of `search_chunk` consecutive bundles (1 .. 8: consecutive bundles
// mostly share a codebook, and every CTA should still get several chunks; striding the chunks
// spreads the tiers, whose bundles differ fourfold in work, evenly over the CTAs); warp = group,
// lane = four token slots.  The only barrier is the codebook change between (head, tier) keys;
// otherwise a warp walks its bundles alone, and while it searches one bundle the page ids and
// source rows of the next are already loaded and its key rows are on their way to L2.
// STAGED: a warp's slices of the next bundle's rows travel to shared memory by 16-byte asynchronous copies, the
// lanes of a row slice side by side, while the current bundle is searched; as one row per lane, every 128-bit
// load fetched 32 sectors and used half of each (GS 16: 106 -> 86 us for a 32768-token prompt).  Chunk c
// of row s is stored at chunk c ^ turn(s), so neither the copies nor the row-per-lane reads meet in a bank.
// Not STAGED: slices off a 16-byte boundary.
// TOK token slots per lane: 4 are a bundle; of few bundles a CTA takes a half or a quarter (blockIdx.y), so that all SMs
// search (see search_parts).
template <int GS, bool STAGED, int TOK>
__global__ void __launch_bounds__(kEncThreads, GS == 16 ? 2 : 1) search_bundles_kernel(const EncodeArgs a) {
  const sphkv_encode_params& p = a.p;
  griddep_wait();
  griddep_launch();
  extern __shared__ __align__(16) uint8_t smem[];
  float* cb_s = reinterpret_cast<float*>(smem);  // [G][C][GS] of the current (head, tier slot)
  const int N = p.page_size, dh = p.dh;
  const int ppb = 128 / N, n_shift = 31 - __clz(N);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = dh / GS, GST = dh >> 4;
  const int esize = p.k_dtype == SPHKV_F32 ? 4 : 2;
  const int chunk_len = a.search_chunk, slot0 = 32 * TOK * blockIdx.y;
  float* scr_r = reinterpret_cast<float*>(p.scratch);
  uint8_t* scr_t = reinterpret_cast<uint8_t*>(p.scratch) + (int64_t)p.n_pages * N * GST * 4;
  // page and source row of this lane's token slots of bundle bi
  auto lookup = [&](int64_t bi, int (&pg)[TOK], int (&row)[TOK]) {
    const int32_t* bundle = p.bundles + 8 * bi;
#pragma unroll
    for (int h = 0; h < TOK; ++h) {
      const int ts = slot0 + lane + 32 * h;
      pg[h] = bundle[ts >> n_shift];
      row[h] = pg[h] >= 0 ? p.src_index[(int64_t)pg[h] * N + (ts & (N - 1))] : -1;
    }
  };
  // 16-byte chunks of a row slice: GS / 4 (fp32) or GS / 8
  const int ch_shift = (GS == 32 ? 3 : 2) - (esize == 2 ? 1 : 0), ch = 1 << ch_shift;
  const uint32_t kbuf = smem_u32(smem + a.search_kbuf) + warp * (32 * TOK * GS * 4);
  auto turn = [&](int s) { return (s >> (3 - ch_shift)) & (ch - 1); };
  auto issue_rows = [&](const int (&row)[TOK], int head) {
    const int s_l = lane >> ch_shift, c = lane & (ch - 1), rows_per = 32 >> ch_shift;
    const char* base = reinterpret_cast<const char*>(p.k_src) + ((int64_t)head * p.k_head_stride + warp * GS) * esize + c * 16;
    const int64_t row_bytes = p.k_row_stride * esize;
#pragma unroll
    for (int h = 0; h < TOK; ++h)
      for (int i = 0; i < ch; ++i) {  // 32 rows, rows_per at a time
        const int s = i * rows_per + s_l;
        const int r = __shfl_sync(0xffffffffu, row[h], s);
        cp_async_16_zfill(kbuf + (((32 * h + s) << ch_shift) + (c ^ turn(s))) * 16, r >= 0 ? base + r * row_bytes : reinterpret_cast<const char*>(p.k_src),
                          r >= 0 ? 16 : 0);
      }
    cp_async_commit();
  };
  int loaded_key = -1;
  for (int64_t chunk = blockIdx.x; chunk * chunk_len < p.n_bundles; chunk += gridDim.x) {
    // lane q < chunk_len looks at bundle q of the chunk: which (head, tier slot), and is it of this
    // launch's group size?  One pair of dependent loads per chunk; bundles of the other group size
    // (the other launch takes them) cost nothing more.
    int my_head = -1, my_slot = 0;
    if (lane < chunk_len && chunk * chunk_len + lane < p.n_bundles) {
      const int32_t* bundle = p.bundles + 8 * (chunk * chunk_len + lane);
      int first = -1;
      for (int q = 0; q < ppb; ++q) {
        const int pq = bundle[q];
        if (first < 0 && pq >= 0) first = pq;
      }
      if (first >= 0) {
        my_head = p.page_head[first];
        my_slot = p.page_slot[first];
      }
    }
    unsigned todo = __ballot_sync(0xffffffffu, my_head >= 0 && p.tiers.g[my_slot] == GS);  // same in every warp
    int pg_n[TOK], row_n[TOK];
    if (todo) {
      lookup(chunk * chunk_len + (__ffs(todo) - 1), pg_n, row_n);
      if (STAGED && warp < G) issue_rows(row_n, __shfl_sync(0xffffffffu, my_head, __ffs(todo) - 1));
    }
    while (todo) {
      const int q = __ffs(todo) - 1;
      todo &= todo - 1;
      const int head = __shfl_sync(0xffffffffu, my_head, q), slot = __shfl_sync(0xffffffffu, my_slot, q);
      int pg[TOK], row[TOK];
#pragma unroll
      for (int h = 0; h < TOK; ++h) { pg[h] = pg_n[h]; row[h] = row_n[h]; }
      int head_n = -1;
      if (todo) {  // the next bundle of the chunk: its rows load while this one is searched
        const int qn = __ffs(todo) - 1;
        head_n = __shfl_sync(0xffffffffu, my_head, qn);
        lookup(chunk * chunk_len + qn, pg_n, row_n);
      }
      if (head * p.tiers.n_slots + slot != loaded_key) {
        __syncthreads();  // every warp is done with the previous codebook
        stage_slot_codebook<GS>(p, head, slot, cb_s);
        loaded_key = head * p.tiers.n_slots + slot;
        __syncthreads();
      }
      if (warp >= G) continue;
      const int bits = p.tiers.bits[slot];
      float k[TOK][GS];
      if (STAGED) {
        cp_async_wait<0>();
        __syncwarp();
#pragma unroll
        for (int h = 0; h < TOK; ++h) {
          const uint32_t src = kbuf + (((32 * h + lane) << ch_shift) * 16);
          if (esize == 4) {
#pragma unroll
            for (int c = 0; c < GS / 4; ++c) {
              const float4 v = lds_f4(src + ((c ^ turn(lane)) << 4));
              k[h][4 * c] = v.x; k[h][4 * c + 1] = v.y; k[h][4 * c + 2] = v.z; k[h][4 * c + 3] = v.w;
            }
          } else {
#pragma unroll
            for (int c = 0; c < GS / 8; ++c) {
              const float4 v = lds_f4(src + ((c ^ turn(lane)) << 4));
              const uint32_t w[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
#pragma unroll
              for (int e = 0; e < 4; ++e) unpack16(w[e], p.k_dtype, k[h][8 * c + 2 * e], k[h][8 * c + 2 * e + 1]);
            }
          }
        }
        __syncwarp();
        if (head_n >= 0) issue_rows(row_n, head_n);
      } else {
        if (head_n >= 0) {
#pragma unroll
          for (int h = 0; h < TOK; ++h)
            if (row_n[h] >= 0)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(
                  reinterpret_cast<const char*>(p.k_src) +
                  ((int64_t)row_n[h] * p.k_row_stride + (int64_t)head_n * p.k_head_stride + warp * GS) * esize));
        }
#pragma unroll
        for (int h = 0; h < TOK; ++h) {
          if (row[h] >= 0) {
            load_group<GS>(p.k_src, p.k_dtype,
                           (int64_t)row[h] * p.k_row_stride + (int64_t)head * p.k_head_stride + warp * GS, k[h]);
          } else {
#pragma unroll
            for (int i = 0; i < GS; ++i) k[h][i] = 0.f;
          }
        }
      }
      float nsq[TOK];
      int code[TOK];
      search_tokens<GS>(k, cb_s + (warp << bits) * GS, 1 << bits, nsq, code);
#pragma unroll
      for (int h = 0; h < TOK; ++h) {
        if (pg[h] < 0) continue;
        const int64_t si = ((int64_t)pg[h] * N + ((slot0 + lane + 32 * h) & (N - 1))) * GST + warp;
        scr_r[si] = row[h] >= 0 ? __fsqrt_rn(nsq[h]) : 0.f;
        scr_t[si] = (uint8_t)code[h];
      }
    }
  }
}

// ---- page assembly, `wpp` warps per page ------------------------------------------------------
// Builds page images from per-(token, group) radii and centroid indices that already exist:
// SRC 2 = the scratch arrays the search launch wrote ([(page * N + slot) * (dh / 16) + group]),
// SRC 3 = a per-token code cache (sphkv_encode_codes) gathered through src_index, i.e. re-paging
// after a tier change without touching the dense keys.  The warps of a page own it from the first lookup
// to the last byte; the only dependent global loads are page index -> src_index row -> code.  16-token
// pages take a warp each (no barrier at all; thousands in flight); a 128-token page is eight warps' work:
// with one, the 440 pages of an 8190-token prompt kept three warps per SM busy (60 us), so 13 us.
// Shared memory of a page: rows i32[N] | r f32[N*G] | scale f32[8] | theta u8[N*G] | page image.
template <int SRC, bool ONE_WARP>
__global__ void __launch_bounds__(kEncThreads) assemble_pages_kernel(const EncodeArgs a) {
  const sphkv_encode_params& p = a.p;
  griddep_wait();
  griddep_launch();
  extern __shared__ __align__(16) uint8_t smem[];
  const int N = p.page_size, dh = p.dh, GST = dh >> 4;
  const int ppb_shift = __clz(N) - 24;  // log2 of the 128 / N pages per bundle (N is 16 .. 128)
  const int wpp_shift = ONE_WARP ? 0 : a.wpp_shift, team = threadIdx.x >> (5 + wpp_shift);
  const int nt = 32 << wpp_shift, t0 = threadIdx.x & (nt - 1), lane = threadIdx.x & 31;  // threads of the page, this one
  const int pages_at_once = (kEncThreads / 32) >> wpp_shift;
  auto page_sync = [&]() {
    if (ONE_WARP)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(nt) : "memory");
  };
  uint8_t* mine = smem + (size_t)team * a.page_smem_bytes;
  int* rows_w = reinterpret_cast<int*>(mine);
  float* r_w = reinterpret_cast<float*>(rows_w + N);
  float* scale_w = r_w + N * GST;
  uint8_t* th_w = reinterpret_cast<uint8_t*>(scale_w + 8);
  uint8_t* img = th_w + N * GST;  // 16-byte aligned: every term above is a multiple of 16
  const float* scr_r = reinterpret_cast<const float*>(p.scratch);
  const uint8_t* scr_t = reinterpret_cast<const uint8_t*>(p.scratch) + (int64_t)p.n_pages * N * GST * 4;
  const int rb = p.radius_fmt == SPHKV_RADIUS_F16 ? 2 : 1;
  const int64_t items = (int64_t)p.n_bundles << ppb_shift;
  for (int64_t it = (int64_t)blockIdx.x * pages_at_once + team; it < items; it += (int64_t)gridDim.x * pages_at_once) {
    const int page = p.bundles[8 * (it >> ppb_shift) + (it & ((1 << ppb_shift) - 1))];
    if (page < 0) continue;
    const int head = p.page_head[page], slot = p.page_slot[page];
    const int64_t poff = p.ptable[3 * (int64_t)page];
    const int gs = p.tiers.g[slot], bits = p.tiers.bits[slot];
    const int G = dh / gs, g_shift = 31 - __clz(G);
    const float* code_r = SRC == 3 ? p.code_r[slot] + (int64_t)head * p.code_rows * G : nullptr;
    const uint8_t* code_t = SRC == 3 ? p.code_theta[slot] + (int64_t)head * p.code_rows * G : nullptr;
    page_sync();  // the previous page's image has been copied out
    // ---- source rows and the valid-token count (valid slots form a prefix); every warp counts all ----
    int cnt = 0;
    for (int s0 = 0; s0 < N; s0 += 32) {
      const int row = s0 + lane < N ? p.src_index[(int64_t)page * N + s0 + lane] : -1;
      if (s0 + lane < N && t0 < 32) rows_w[s0 + lane] = row;
      cnt += __popc(__ballot_sync(0xffffffffu, row >= 0));
    }
    if (!ONE_WARP && t0 < 8) scale_w[t0] = 0.f;
    page_sync();
    // ---- radii and centroid indices of the page; per-group scale = max radius over its tokens.  A thread's
    //      items all belong to one group (32 is a multiple of G) ----
    {
      float mx = 0.f;
#pragma unroll 4
      for (int i = t0; i < N * G; i += nt) {
        const int tin = i >> g_shift, gq = i & (G - 1);
        float rv = 0.f;
        uint8_t tv = 0;
        if (SRC == 2) {
          const int64_t si = ((int64_t)page * N + tin) * GST + gq;
          rv = scr_r[si];
          tv = scr_t[si];
        } else {
          const int row = rows_w[tin];
          if (row >= 0) {
            rv = code_r[(int64_t)row * G + gq];
            tv = code_t[(int64_t)row * G + gq];
          }
        }
        r_w[i] = rv;
        th_w[i] = tv;
        if (tin < cnt) mx = fmaxf(mx, rv);
      }
      for (int o = G; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane < G) {
        if (ONE_WARP)
          scale_w[lane] = mx;
        else  // radii are not negative: their bit patterns order as integers
          atomicMax(reinterpret_cast<int*>(scale_w + lane), __float_as_int(mx));
      }
    }
    page_sync();
    if (cnt > 0) {
      // ---- header, scales, LSB-first theta words ----------------------------------------------
      const int hdr = 8 + 4 * G;
      const int nvals = cnt * G;
      const int th_bytes = (nvals * bits + 7) >> 3;
      const int th_words = (th_bytes + 3) >> 2;
      if (t0 < 2)
        reinterpret_cast<uint32_t*>(img)[t0] =
            t0 == 0 ? (uint32_t)(p.tiers.tier_id[slot] & 0xFF) | ((uint32_t)(cnt & 0xFF) << 8) |
                          ((uint32_t)(p.radius_fmt & 0xFF) << 16)
                    : 0u;
      if (t0 < G) reinterpret_cast<float*>(img + 8)[t0] = scale_w[t0];
      for (int w = t0; w < th_words; w += nt) {
        const int bit0 = w * 32;
        const int i0 = bit0 / bits;                             // first value overlapping this word
        const int i1 = min(nvals, (bit0 + 31) / bits + 1);      // one past the last
        // values enter a 64-bit window that starts 8 bits below the word, so a value that begins
        // in the previous word (bits <= 8) needs no right shift
        int sh = i0 * bits - bit0 + 8;
        unsigned long long acc = 0;
        for (int i = i0; i < i1; ++i, sh += bits) acc |= (unsigned long long)th_w[i] << sh;
        reinterpret_cast<uint32_t*>(img + hdr)[w] = (uint32_t)(acc >> 8);
      }
      page_sync();
      // ---- radii (may overlay the zero tail of the last theta word) ---------------------------
      uint8_t* rad = img + hdr + th_bytes;
      for (int i = t0; i < nvals; i += nt) {
        const float rr = r_w[i];
        if (rb == 1) {
          const float safe = fmaxf(scale_w[i & (G - 1)], 1e-8f);
          float qv = rintf(__fmul_rn(__fdiv_rn(rr, safe), 127.0f));
          qv = fminf(fmaxf(qv, -127.f), 127.f);
          rad[i] = (uint8_t)(int8_t)(int)qv;
        } else {
          // the half's bit pattern goes over the radius slot as a 32-bit word (this thread read it
          // just above); its two bytes are laid into the image below
          reinterpret_cast<uint32_t*>(r_w)[i] = (uint32_t)__half_as_ushort(__float2half_rn(rr));
        }
      }
      page_sync();
      if (rb == 2) {
        const uint8_t* hb = reinterpret_cast<const uint8_t*>(r_w);
        for (int b2 = t0; b2 < 2 * nvals; b2 += nt) rad[b2] = hb[(b2 >> 1) * 4 + (b2 & 1)];
        page_sync();
      }
      // ---- copy the image out ----------------------------------------------------------------
      const int bytes = hdr + th_bytes + nvals * rb;
      for (int w = t0; w < (bytes >> 2); w += nt)
        reinterpret_cast<uint32_t*>(p.k_pages + poff)[w] = reinterpret_cast<const uint32_t*>(img)[w];
      if (t0 < (bytes & 3)) p.k_pages[poff + (bytes & ~3) + t0] = img[(bytes & ~3) + t0];
    }
    // ---- dense V page (16-bit), empty slots zero-filled; four chunks in flight per thread -------
    if (p.v_src != nullptr && p.v_pool != nullptr) {
      constexpr int kInFlight = 4;
      const int pr_shift = 31 - __clz(dh >> 3);  // 16-byte chunks per row (dh / 8, a power of two)
      const bool same = p.v_src_dtype == p.v_pool_dtype;
      const int chunks = N << pr_shift;
      for (int i0 = t0; i0 < chunks; i0 += nt * kInFlight) {
        uint4 o[kInFlight];
#pragma unroll
        for (int e = 0; e < kInFlight; ++e) {
          const int i = i0 + e * nt;
          o[e] = make_uint4(0u, 0u, 0u, 0u);
          if (i >= chunks) continue;
          const int tin = i >> pr_shift, d = (i & ((1 << pr_shift) - 1)) * 8;
          const int row = rows_w[tin];
          if (row >= 0) o[e] = load_v_chunk(p, same, (int64_t)row * p.v_row_stride + (int64_t)head * p.v_head_stride + d);
        }
#pragma unroll
        for (int e = 0; e < kInFlight; ++e)
          if (i0 + e * nt < chunks)
            reinterpret_cast<uint4*>(p.v_pool)[(((int64_t)page * N * dh) >> 3) + i0 + e * nt] = o[e];
      }
    }
  }
}

// ---- all-tier code cache ---------------------------------------------------------------------
// Radius and nearest centroid of every (token, KV head, group) for EVERY tier slot in one pass
// over the keys (the pre-encode of spherical_kv_pipeline.py:1535-1553, which calls
// _encode_keys_with_codebooks once per tier).  Output per slot s, head-major like the
// reference's per-(layer, head) cache: r[s][head][row][G_s] f32, theta[s][head][row][G_s] u8.
struct ChainArgs {
  const void* k_src;
  const float* codebooks;
  float* r_out[SPHKV_MAX_TIER_SLOTS];
  uint8_t* th_out[SPHKV_MAX_TIER_SLOTS];
  int64_t k_row_stride, k_head_stride, rows;
  int64_t n_units, units_per_head;  // unit = one CTA pass: (8 / (dh / 32)) * 32 * kCodeTok rows of one head
  int k_dtype, dh;
  int kbuf_off;  // byte offset of the staged row blocks (8 warps x 32 * kCodeTok rows x 128 B)
  int cb_off[SPHKV_MAX_TIER_SLOTS];  // float offset of each slot's staged codebook
  sphkv_tiers tiers;
};

template <int OFF, int GS, int kCodeTok>
__device__ __forceinline__ void search_slice(const float (&k)[kCodeTok][32], const float* __restrict__ cbg, int C,
                                             int (&code)[kCodeTok]) {
  float best[kCodeTok];
#pragma unroll
  for (int h = 0; h < kCodeTok; ++h) { best[h] = -INFINITY; code[h] = 0; }
  SPHKV_UNROLL_CODE_SEARCH
  for (int c = 0; c < C; ++c) {
    const float4* row = reinterpret_cast<const float4*>(cbg + c * GS);
    float sacc[kCodeTok];
#pragma unroll
    for (int h = 0; h < kCodeTok; ++h) sacc[h] = 0.f;
#pragma unroll
    for (int i = 0; i < GS / 4; ++i) {
      const float4 v = row[i];
#pragma unroll
      for (int h = 0; h < kCodeTok; ++h) {
        sacc[h] = __fmaf_rn(k[h][OFF + 4 * i], v.x, sacc[h]);
        sacc[h] = __fmaf_rn(k[h][OFF + 4 * i + 1], v.y, sacc[h]);
        sacc[h] = __fmaf_rn(k[h][OFF + 4 * i + 2], v.z, sacc[h]);
        sacc[h] = __fmaf_rn(k[h][OFF + 4 * i + 3], v.w, sacc[h]);
      }
    }
#pragma unroll
    for (int h = 0; h < kCodeTok; ++h)
      if (sacc[h] > best[h]) { best[h] = sacc[h]; code[h] = c; }
  }
}

#ifndef SPHKV_CODE_WARPS
#define SPHKV_CODE_WARPS 8
#endif
constexpr int kChainThreads = SPHKV_CODE_WARPS * 32;  // a multiple of four warps: dh / 32 warps share a token set

// Few centroids, short inputs (see the rule at the launch): the chains on the fp32 pipe.  A thread holds four tokens' 32-dim slice; the two
// 16-dim halves serve the g = 16 tiers, the whole slice the g = 32 tiers, and the squared norm of the 32-dim group
// continues the fma chain of its first half, so every value equals what the per-tier encoder computes.
// Persistent: the (head, row block) units are dealt out in contiguous runs, one run per resident
// CTA.  A CTA stages a head's codebooks when its run enters that head (once or twice per CTA) and
// has no other barrier, so the warps of an SM drift apart and one warp's key loads hide under the
// others' searches.  STAGED: a warp's next row block travels global -> shared memory by 16-byte
// asynchronous copies (eight lanes per 128-byte row slice, so every sector is used whole) while
// the current block is searched; the chunk index is XOR-ed with the row so that both the copies
// and the later one-row-per-lane 128-bit reads touch every bank once.  Not STAGED (slices not
// 16-byte aligned, or no room beside the codebooks): each lane loads its own rows and asks L2
// for the next block's rows a block ahead.
// kCodeTok tokens per thread: four feed 16 fmas from every centroid load (232 registers); with two or one a small
// input reaches more SMs and waits for a shorter pass (419 tokens x 8 heads: 27 -> 14 us; 2048: 27 -> 19).
template <bool STAGED, int kCodeTok>
__global__ void __launch_bounds__(kChainThreads, 1) codes_chains_kernel(const ChainArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  float* cb_s = reinterpret_cast<float*>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G32 = a.dh >> 5;                  // 32-dim groups per head: 2 or 4
  const int grp = warp % G32, set = warp / G32;
  const int sets = (kChainThreads / 32) / G32;  // token sets of 32 * kCodeTok per CTA
  constexpr int kBlockRows = 32 * kCodeTok;
  const int esize = a.k_dtype == SPHKV_F32 ? 4 : 2;
  const int64_t u_lo = a.n_units * blockIdx.x / gridDim.x, u_hi = a.n_units * (blockIdx.x + 1) / gridDim.x;
  const bool k32 = a.k_dtype == SPHKV_F32;
  const uint32_t kbuf = smem_u32(smem + a.kbuf_off) + warp * (kBlockRows * 128);  // this warp's row block
  auto issue_block = [&](int64_t uu) {
    const int64_t hd = uu / a.units_per_head;
    const int64_t c0 = hd * a.k_head_stride + grp * 32;
    const int64_t r0 = ((uu - hd * a.units_per_head) * sets + set) * kBlockRows;
    // lane -> (row lane / CH, chunk lane % CH) of every group of 32 / CH rows; one pointer walks the rows
    const int esz = k32 ? 4 : 2, ch_shift = k32 ? 3 : 2, rows_per_i = 32 >> ch_shift;
    const int r_l = lane >> ch_shift, c = lane & ((1 << ch_shift) - 1);
    // chunk swizzle: row & 7 for 128-byte rows, (row >> 1) & 3 for 64-byte rows.  Eight 64-byte rows
    // per step keep it fixed; four 128-byte rows per step flip bit 2 of it on odd steps.
    const int sw = k32 ? r_l : ((r_l >> 1) & 3);
    const char* src = reinterpret_cast<const char*>(a.k_src) + ((r0 + r_l) * a.k_row_stride + c0) * esz + c * 16;
    const int64_t src_step = a.k_row_stride * esz * rows_per_i;
    const uint32_t dst = kbuf + ((r_l << ch_shift) + (c ^ sw)) * 16;
    const uint32_t dst_odd = k32 ? kbuf + ((r_l << ch_shift) + (c ^ sw ^ 4)) * 16 : dst;
    const int64_t left = a.rows - r0 - r_l;  // rows of the block at or below this lane's first one
    if (left >= kBlockRows) {
#pragma unroll
      for (int i = 0; i < kBlockRows / 4; ++i) {
        if (i < kBlockRows / rows_per_i) cp_async_16(((i & 1) ? dst_odd : dst) + i * 512, src + i * src_step);
      }
    } else {
#pragma unroll
      for (int i = 0; i < kBlockRows / 4; ++i) {
        if (i < kBlockRows / rows_per_i) {
          const bool in = (int64_t)i * rows_per_i < left;
          cp_async_16_zfill(((i & 1) ? dst_odd : dst) + i * 512, in ? src + i * src_step : reinterpret_cast<const char*>(a.k_src), in ? 16 : 0);
        }
      }
    }
    cp_async_commit();
  };
  if (STAGED && u_lo < u_hi) issue_block(u_lo);
  int head = -1;
  for (int64_t u = u_lo; u < u_hi; ++u) {
    const int u_head = (int)(u / a.units_per_head);
    if (u_head != head) {
      // stage every slot's codebook of this head: [G_s][C_s][g_s] packed
      if (head >= 0) __syncthreads();
      head = u_head;
      for (int s = 0; s < a.tiers.n_slots; ++s) {
        const int gs = a.tiers.g[s], bits = a.tiers.bits[s], G = a.dh / gs, q4n = gs >> 2;
        const float4* src = reinterpret_cast<const float4*>(
            a.codebooks + ((int64_t)(head * a.tiers.n_slots + s) * a.tiers.G_max) * a.tiers.C_max * a.tiers.g_max);
        float4* dst = reinterpret_cast<float4*>(cb_s + a.cb_off[s]);
        const int total = (G << bits) * q4n, row_stride4 = a.tiers.g_max >> 2;
        for (int i = threadIdx.x; i < total; i += blockDim.x) {
          const int q4 = i % q4n, row = i / q4n;
          dst[i] = __ldg(src + ((int64_t)(row >> bits) * a.tiers.C_max + (row & ((1 << bits) - 1))) * row_stride4 + q4);
        }
      }
      __syncthreads();
    }
    const int64_t col = (int64_t)head * a.k_head_stride + grp * 32;
    const int64_t row0 = ((u - (int64_t)head * a.units_per_head) * sets + set) * kBlockRows;
    if (!STAGED && u + 1 < u_hi) {
      const int64_t ncol = (u + 1) / a.units_per_head * a.k_head_stride + grp * 32;
      const int64_t nrow0 = ((u + 1) % a.units_per_head * sets + set) * kBlockRows;
#pragma unroll
      for (int h = 0; h < kCodeTok; ++h) {
        const int64_t nrow = nrow0 + lane + 32 * h;
        if (nrow < a.rows)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(a.k_src) + (nrow * a.k_row_stride + ncol) * esize));
      }
    }
    float k[kCodeTok][32];
    bool have[kCodeTok];
    if (STAGED) {
      cp_async_wait<0>();
      __syncwarp();
#pragma unroll
      for (int h = 0; h < kCodeTok; ++h) {
        have[h] = row0 + lane + 32 * h < a.rows;
        const int r = h * 32 + lane;
        if (k32) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float4 v = lds_f4(kbuf + r * 128 + ((c ^ (lane & 7)) << 4));
            k[h][4 * c] = v.x; k[h][4 * c + 1] = v.y; k[h][4 * c + 2] = v.z; k[h][4 * c + 3] = v.w;
          }
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float4 v = lds_f4(kbuf + r * 64 + ((c ^ ((lane >> 1) & 3)) << 4));
            const uint32_t w[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
#pragma unroll
            for (int e = 0; e < 4; ++e) unpack16(w[e], a.k_dtype, k[h][8 * c + 2 * e], k[h][8 * c + 2 * e + 1]);
          }
        }
      }
      __syncwarp();
      if (u + 1 < u_hi) issue_block(u + 1);
    } else
#pragma unroll
    for (int h = 0; h < kCodeTok; ++h) {
      const int64_t row = row0 + lane + 32 * h;
      have[h] = row < a.rows;
      if (have[h]) {
        load_group<32>(a.k_src, a.k_dtype, row * a.k_row_stride + col, k[h]);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) k[h][i] = 0.f;
      }
    }
    float na[kCodeTok], nb[kCodeTok], nab[kCodeTok];
#pragma unroll
    for (int h = 0; h < kCodeTok; ++h) na[h] = nb[h] = 0.f;
#pragma unroll
    for (int d = 0; d < 16; ++d)
#pragma unroll
      for (int h = 0; h < kCodeTok; ++h) {
        na[h] = __fmaf_rn(k[h][d], k[h][d], na[h]);
        nb[h] = __fmaf_rn(k[h][16 + d], k[h][16 + d], nb[h]);
      }
#pragma unroll
    for (int h = 0; h < kCodeTok; ++h) nab[h] = na[h];
#pragma unroll
    for (int d = 16; d < 32; ++d)
#pragma unroll
      for (int h = 0; h < kCodeTok; ++h) nab[h] = __fmaf_rn(k[h][d], k[h][d], nab[h]);

    for (int s = 0; s < a.tiers.n_slots; ++s) {
      if (a.r_out[s] == nullptr) continue;
      const int bits = a.tiers.bits[s], C = 1 << bits;
      if (a.tiers.g[s] == 16) {
        // both 16-dim halves of the slice, stored as one 8-byte radius pair and one 2-byte code pair
        const int G = a.dh >> 4;
        int code_a[kCodeTok], code_b[kCodeTok];
        search_slice<0, 16, kCodeTok>(k, cb_s + a.cb_off[s] + ((2 * grp) << bits) * 16, C, code_a);
        search_slice<16, 16, kCodeTok>(k, cb_s + a.cb_off[s] + ((2 * grp + 1) << bits) * 16, C, code_b);
#pragma unroll
        for (int h = 0; h < kCodeTok; ++h) {
          if (!have[h]) continue;
          const int64_t o = ((int64_t)head * a.rows + row0 + lane + 32 * h) * G + 2 * grp;
          *reinterpret_cast<float2*>(a.r_out[s] + o) = make_float2(__fsqrt_rn(na[h]), __fsqrt_rn(nb[h]));
          *reinterpret_cast<uint16_t*>(a.th_out[s] + o) = (uint16_t)(code_a[h] | (code_b[h] << 8));
        }
      } else {
        int code[kCodeTok];
        search_slice<0, 32, kCodeTok>(k, cb_s + a.cb_off[s] + (grp << bits) * 32, C, code);
#pragma unroll
        for (int h = 0; h < kCodeTok; ++h) {
          if (!have[h]) continue;
          const int64_t o = ((int64_t)head * a.rows + row0 + lane + 32 * h) * G32 + grp;
          a.r_out[s][o] = __fsqrt_rn(nab[h]);
          a.th_out[s][o] = (uint8_t)code[h];
        }
      }
    }
  }
}

// ---- the same on the tensor cores ----
struct CodesArgs {
  const void* k_src;
  const float* codebooks;
  float* r_out[SPHKV_MAX_TIER_SLOTS];
  uint8_t* th_out[SPHKV_MAX_TIER_SLOTS];
  int64_t k_row_stride, k_head_stride, rows;
  int64_t n_units, units_per_head;  // unit = 128 rows of one head
  int k_dtype, dh;
  int kbuf_off;  // byte offset of the staged rows
  int wide;      // outputs start on 16 (r) and 4 bytes (theta)
  sphkv_tiers tiers;
  SearchPlan plan;
};

// Row slices of 32 dims wait in shared memory, 128 (fp32) or 64 bytes a row, a 4 KB block per warp and stage; chunk c of
// row r is stored at chunk c ^ (r & 7), or c ^ (r >> 1 & 3): neither the copies (the lanes of a row side by side) nor
// the row-per-lane reads meet in a bank.
constexpr int kSliceBlock = 4096;
__device__ __forceinline__ int staged_chunk(bool k32, int r, int c) { return k32 ? c ^ (r & 7) : c ^ ((r >> 1) & 3); }
__device__ __forceinline__ void read_staged_row(uint32_t block, int dtype, float (&k)[32]) {
  const int lane = threadIdx.x & 31;
  if (dtype == SPHKV_F32) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float4 v = lds_f4(block + lane * 128 + (staged_chunk(true, lane, c) << 4));
      k[4 * c] = v.x; k[4 * c + 1] = v.y; k[4 * c + 2] = v.z; k[4 * c + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 v = lds_f4(block + lane * 64 + (staged_chunk(false, lane, c) << 4));
      const uint32_t x[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
#pragma unroll
      for (int e = 0; e < 4; ++e) unpack16(x[e], dtype, k[8 * c + 2 * e], k[8 * c + 2 * e + 1]);
    }
  }
}
__device__ __forceinline__ void group_barrier(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kSearchWarps * 32) : "memory");
}
// `count` (1, 2 or 4) neighbouring radii and codes (a byte each); 16- and 4-byte stores where `wide`
__device__ __forceinline__ void store_groups(float* r, uint8_t* theta, int count, bool wide, float4 v, uint32_t codes) {
  if (count == 4 && wide) {
    *reinterpret_cast<float4*>(r) = v;
    *reinterpret_cast<uint32_t*>(theta) = codes;
  } else if (count >= 2) {
    *reinterpret_cast<float2*>(r) = make_float2(v.x, v.y);
    *reinterpret_cast<uint16_t*>(theta) = (uint16_t)codes;
    if (count == 4) {
      *reinterpret_cast<float2*>(r + 2) = make_float2(v.z, v.w);
      *reinterpret_cast<uint16_t*>(theta + 2) = (uint16_t)(codes >> 16);
    }
  } else {
    *r = v.x;
    *theta = (uint8_t)codes;
  }
}

// The fma chains' answer for the lanes in `open`: group `gamma` of key row `row`; kFirstWins (low byte 0) for a vector of zeros, or
// with a NaN, where many lanes are open.  Bound by what it reads: keys and centroids come from L2, row by row.  32768 tokens x 8 heads,
// three tiers, by the data (every lane walking all centroids of an open search before / now / the chains' kernel): random 76 / 77 / 170
// us; a third of the keys' mean as spread 124 / 114 / 170, a tenth 396 / 227 / 170; zeros 870 / 140 / 174; every search a tie
// 865 / 790 / 170.  Columns instead of lanes (as k-means does) take registers that the searches need: 81 to 92 us for random keys.
constexpr int kFirstWins = 256;
template <int GS>
__device__ __noinline__ int settle(const CodesArgs& p, int head, int s, int gamma, int64_t row, unsigned open, int code) {
  const sphkv_tiers& t = p.tiers;
  const float* cb = p.codebooks + (((int64_t)(head * t.n_slots + s) * t.G_max + gamma) * t.C_max) * t.g_max;
  float k[GS];
  if ((open >> (threadIdx.x & 31)) & 1u) {
    load_group<GS>(p.k_src, p.k_dtype, row * p.k_row_stride + (int64_t)head * p.k_head_stride + gamma * GS, k);
  } else {
#pragma unroll
    for (int d = 0; d < GS; ++d) k[d] = 0.f;
  }
  if (__popc(open) > 4) {
    const bool first = ((open >> (threadIdx.x & 31)) & 1u) && first_wins(k, cb);
    if (first) code = kFirstWins;
    open &= ~__ballot_sync(0xffffffffu, first);
    if (open == 0) return code;
  }
  return exact_search(k, cb, t.g_max, 1 << t.bits[s], open, code);
}

constexpr int kCodeStages = 4;                                  // slices in flight

constexpr int kCodeTail = 256;  // norms, barriers, tensor memory base

// A set of tiers that the kernel below is compiled for: centroid bits of two 16-dim slots and one 32-dim slot (0: none),
// in that order.  Its sums are a slice's columns [16-dim slots | the same, second half | 32-dim slot], all loaded at once.
template <int B0, int B1, int B2>
struct FixedTiers {
  static constexpr bool kFixed = B0 > 0;
  static constexpr int kSlots = (B0 > 0) + (B1 > 0) + (B2 > 0);
  static constexpr int C0 = B0 ? 1 << B0 : 0, C1 = B1 ? 1 << B1 : 0, C2 = B2 ? 1 << B2 : 0;
  static constexpr int kHalf = (C0 + C1 + 15) / 16 * 16;  // columns of a half
  static bool match(const sphkv_tiers& t, unsigned wanted) {
    if (!kFixed || t.n_slots != kSlots || wanted != (1u << kSlots) - 1) return false;
    const int bits[3] = {B0, B1, B2}, g[3] = {16, 16, 32};
    for (int s = 0; s < kSlots; ++s)
      if (t.bits[s] != bits[s] || t.g[s] != g[s]) return false;
    return true;
  }
};
using AnyTiers = FixedTiers<0, 0, 0>;

// Persistent: the (head, 128-row block) units are dealt out in contiguous runs, one run per CTA; a CTA lays a head's
// centroids out for the tensor cores when its run enters that head.  Its two search groups share every unit: each takes
// half of the 32-dim slices, so the groups never wait for one another between heads and small inputs spread over
// more SMs.  Thread = row = lane of tensor memory; slice by slice: the sums into registers, so that the tensor cores can
// multiply the next slice at once; their searches; the slice after that from shared memory, its norms' fma chains, its
// bf16 pairs to tensor memory.  STAGED: rows travel global -> shared memory by 16-byte asynchronous copies four slices
// ahead.  Not STAGED (slices off a 16-byte boundary, or no room beside the centroids): each lane loads its own row.
// AnyTiers: slots of any number and size, in passes of what fits, branch by branch; the instructions around the searches are
// then as many as those of the searches.
template <bool STAGED, typename Fix>
__global__ void __launch_bounds__(kSearchThreads, 1) encode_codes_kernel(const __grid_constant__ CodesArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int group = warp / kSearchWarps, w = warp % kSearchWarps;
  float* most = reinterpret_cast<float*>(smem + a.plan.bytes);
  const uint32_t bars = smem_u32(smem + a.plan.bytes + 128), bar = bars + 8 * group;
  volatile uint32_t* tmem_word = reinterpret_cast<volatile uint32_t*>(smem + a.plan.bytes + 128 + 8 * kSearchGroups);
  if (warp == 0) tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_word)), kSearchGroups * kGroupCols);
  if (threadIdx.x < kSearchGroups) mbar_init(bars + 8 * threadIdx.x, 1);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_word[0], 0);
  const uint32_t tmem = tmem_base + group * kGroupCols, my_rows = tmem + ((uint32_t)(32 * w) << 16);

  const int64_t u_lo = a.n_units * blockIdx.x / gridDim.x, u_hi = a.n_units * (blockIdx.x + 1) / gridDim.x;
  const int per = a.dh / 32 / kSearchGroups;   // slices of this group: 1 or 2
  const int slice0 = group * per;
  const int n_q = (int)(u_hi - u_lo) * per;    // (unit, slice) pairs this group walks
  const bool k32 = a.k_dtype == SPHKV_F32, lows = a.k_dtype != SPHKV_BF16;
  const int esz = k32 ? 4 : 2, ch_shift = k32 ? 3 : 2;  // 16-byte chunks of a row slice: 8 or 4
  // Where a (unit, slice) pair lies.  Three of these walk the pairs: rows are fetched kCodeStages pairs ahead of the split,
  // which is two pairs ahead of the search (dividing for each cost a third of the kernel's instructions).
  struct Place {
    int q, slice, head;
    int64_t row0;  // first row of the warp's 32
  };
  Place at0;
  at0.q = 0;
  at0.slice = slice0;
  at0.head = (int)(u_lo / a.units_per_head);
  at0.row0 = (u_lo - at0.head * a.units_per_head) * 128 + 32 * w;
  const int64_t head_rows = a.units_per_head * 128;
  auto advance = [&](Place& p) {
    ++p.q;
    if (++p.slice < slice0 + per) return;
    p.slice = slice0;
    p.row0 += 128;
    if (p.row0 >= head_rows) {
      p.row0 -= head_rows;
      ++p.head;
    }
  };
  const uint32_t kbuf = smem_u32(smem + a.kbuf_off) + warp * (kCodeStages * kSliceBlock);
  Place fetch = at0;
  const int r_l = lane >> ch_shift, c_l = lane & ((1 << ch_shift) - 1);  // this lane's first row of a block, its chunk
  const int64_t row_bytes = a.k_row_stride * esz, src_step = row_bytes * (32 >> ch_shift);
  auto fetch_base = [&]() {
    return reinterpret_cast<const char*>(a.k_src) + (fetch.row0 + r_l) * row_bytes + ((int64_t)fetch.head * a.k_head_stride + fetch.slice * 32) * esz +
           c_l * 16;
  };
  const char* fetch_src = fetch_base();
  // (four 128-byte rows a step flip bit 2 of the chunk on odd steps, eight 64-byte rows do not)
  const uint32_t to_even = ((r_l << ch_shift) + staged_chunk(k32, r_l, c_l)) * 16, to_odd = k32 ? to_even ^ 64 : to_even;
  auto issue_rows = [&]() {
    if (fetch.q < n_q) {
      const uint32_t dst = kbuf + (fetch.q & (kCodeStages - 1)) * kSliceBlock;
      const char* src = fetch_src;
      if (a.rows - fetch.row0 >= 32) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i < 4 || k32) cp_async_16(dst + ((i & 1) ? to_odd : to_even) + i * 512, src);
          src += src_step;
        }
      } else {
        const int left = (int)max((int64_t)-64, a.rows - fetch.row0) - r_l;  // rows from this lane's first on
        for (int i = 0; i < (1 << ch_shift); ++i) {
          const bool in = (i << (5 - ch_shift)) < left;
          cp_async_16_zfill(dst + ((i & 1) ? to_odd : to_even) + i * 512, in ? src : reinterpret_cast<const char*>(a.k_src), in ? 16 : 0);
          src += src_step;
        }
      }
      const int head = fetch.head, slice = fetch.slice;
      advance(fetch);
      fetch_src = fetch.head != head ? fetch_base() : fetch_src + (fetch.slice - slice) * 32 * esz + (fetch.slice <= slice ? 128 * row_bytes : 0);
    }
    cp_async_commit();
  };

  Place next = at0;
  auto convert = [&]() -> SliceNorms {  // the pair `next`
    float k[32];
    if (STAGED) {
      cp_async_wait<kCodeStages - 1>();
      __syncwarp();
      read_staged_row(kbuf + (next.q & (kCodeStages - 1)) * kSliceBlock, a.k_dtype, k);
      __syncwarp();
      issue_rows();
    } else if (next.row0 + lane < a.rows) {
      load_group<32>(a.k_src, a.k_dtype, (next.row0 + lane) * a.k_row_stride + (int64_t)next.head * a.k_head_stride + next.slice * 32, k);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) k[i] = 0.f;
    }
    const SliceNorms nn = store_slice(k, my_rows + kKeyCols + (next.q & 1) * 32, lows);
    advance(next);
    return nn;
  };
  const uint32_t op = smem_u32(smem);
  Place cur = at0;
  ProductWaits waits;  // once one ran out the chains decide everything
  auto wait = [&](uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0; };
  auto products = [&](int ps) {  // of the pair `cur`, by the group's first warp, after the group's barrier
    if (w != 0 || waits.lost) return;
    tc_fence_after();
    if (elect_one()) {
      const uint32_t keys = tmem + kKeyCols + (cur.q & 1) * 32;
      if constexpr (Fix::kFixed) {
        constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);  // fp32 sums, bf16 x bf16, 128 rows
        constexpr uint32_t k16 = kIdesc | (Fix::kHalf / 8) << 17, k32 = kIdesc | 2u << 17;
        constexpr uint32_t kRows = 2 * Fix::kHalf + (Fix::C2 ? 32 : 0), kLo = kRows * 2;  // operand rows of a part; 16-byte units
        const uint64_t b = smem_desc(op, 128, 256, 0) + (uint32_t)(cur.slice * 2 * kRows * 2);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint64_t hi = b + half * Fix::kHalf * 2;
          const uint32_t d = tmem + half * Fix::kHalf;
          mma_ts(d, keys + 8 * half, hi, k16, false);
          if (lows) mma_ts(d, keys + 16 + 8 * half, hi, k16, true);
          mma_ts(d, keys + 8 * half, hi + kLo, k16, true);
          if (lows) mma_ts(d, keys + 16 + 8 * half, hi + kLo, k16, true);
        }
        if constexpr (Fix::C2 > 0) {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const uint64_t hi = b + (2 * Fix::kHalf + 16 * half) * 2;
            const uint32_t d = tmem + 2 * Fix::kHalf;
            mma_ts(d, keys + 8 * half, hi, k32, half > 0);
            if (lows) mma_ts(d, keys + 16 + 8 * half, hi, k32, true);
            mma_ts(d, keys + 8 * half, hi + kLo, k32, true);
            if (lows) mma_ts(d, keys + 16 + 8 * half, hi + kLo, k32, true);
          }
        }
      } else {
        issue_products(a.plan, a.tiers, ps, tmem, keys, op + a.plan.base[ps] + cur.slice * 2 * a.plan.rows[ps] * 32, lows);
      }
      mma_commit(bar);
    }
    __syncwarp();
  };
  auto enter_head = [&](int head) {  // between barriers of the whole CTA
    stage_centroids(a.plan, a.tiers, a.codebooks, head, a.dh, smem, most);
  };

  if (n_q > 0) {
    if (STAGED)
      for (int i = 0; i < kCodeStages; ++i) issue_rows();
    int head_at = cur.head;
    enter_head(head_at);
    SliceNorms n0 = convert(), n1 = {};  // of the pair that is searched next, and of the one after
    if (next.q < n_q) n1 = convert();
    tc_fence_before();
    __syncthreads();
    products(0);
    uint32_t codes_before[3] = {0, 0, 0};
    SliceNorms before = {};
    for (int ps = 0;;) {
      const bool last_pass = Fix::kFixed || ps + 1 == a.plan.n_pass;
      waits.next(wait);
      const bool lost = waits.lost;
      tc_fence_after();
      const int slice = cur.slice, head = cur.head;
      const int64_t row = cur.row0 + lane;
      const bool have = row < a.rows;
      constexpr int kC0 = Fix::kFixed ? Fix::C0 : 16, kC1 = Fix::C1 ? Fix::C1 : 16, kC2 = Fix::C2 ? Fix::C2 : 16;
      float s0a[kC0 < 16 ? 16 : kC0], s0b[kC0 < 16 ? 16 : kC0], s1a[kC1 < 16 ? 16 : kC1], s1b[kC1 < 16 ? 16 : kC1], s2[kC2 < 16 ? 16 : kC2];
      float2 far0 = {}, far1 = {};
      float far2 = 0.f;
      if constexpr (Fix::kFixed) {
        tmem_ld_row<kC0>(my_rows, s0a);
        tmem_ld_row<kC0>(my_rows + Fix::kHalf, s0b);
        far0 = *reinterpret_cast<const float2*>(most + 2 * slice);
        if constexpr (Fix::C1 > 0) {
          tmem_ld_row<kC1>(my_rows + Fix::C0, s1a);
          tmem_ld_row<kC1>(my_rows + Fix::kHalf + Fix::C0, s1b);
          far1 = *reinterpret_cast<const float2*>(most + 8 + 2 * slice);
        }
        if constexpr (Fix::C2 > 0) {
          tmem_ld_row<kC2>(my_rows + 2 * Fix::kHalf, s2);
          far2 = most[8 * (Fix::kSlots - 1) + slice];
        }
        tmem_wait_ld();
      } else {
        for (int li = a.plan.first[ps]; li < a.plan.first[ps + 1]; ++li) {
          const int s = a.plan.list[li], bits = a.tiers.bits[s];
          const bool two = a.tiers.g[s] == 16;
          const uint32_t sums = my_rows + a.plan.col[s];
          RowSums v;
          load_sums(v, sums, sums + a.plan.n16[ps], bits, two);
          int ca, cb;
          bool sa, sb;
          search_sums(v, bits, two, two ? n0.a : n0.ab, n0.b, most[s * 8 + (two ? 2 * slice : slice)], most[s * 8 + (two ? 2 * slice + 1 : 0)], ca, cb, sa, sb);
          if (__any_sync(0xffffffffu, have && (lost || !(sa && sb)))) {
            const unsigned open_a = __ballot_sync(0xffffffffu, have && (lost || !sa)), open_b = __ballot_sync(0xffffffffu, have && (lost || !sb));
            if (two) {
              if (open_a) ca = settle<16>(a, head, s, 2 * slice, row, open_a, ca) & 255;
              if (open_b) cb = settle<16>(a, head, s, 2 * slice + 1, row, open_b, cb) & 255;
            } else {
              ca = settle<32>(a, head, s, slice, row, open_a, ca) & 255;
            }
          }
          if (have) {
            const int G = two ? a.dh >> 4 : a.dh >> 5;
            const int64_t o = ((int64_t)head * a.rows + row) * G + (two ? 2 * slice : slice);
            store_groups(a.r_out[s] + o, a.th_out[s] + o, two ? 2 : 1, false, two ? make_float4(n0.a, n0.b, 0.f, 0.f) : make_float4(n0.ab, 0.f, 0.f, 0.f),
                         two ? ca | (cb << 8) : ca);
          }
        }
      }
      // the sums have been read: the next products
      tc_fence_before();
      ++ps;
      if (last_pass) {
        advance(cur);
        ps = 0;
      }
      const bool more = cur.q < n_q;
      if (more) {
        if (cur.head != head_at) {  // both groups walk the same units, so they meet here
          head_at = cur.head;
          __syncthreads();
          enter_head(head_at);
          __syncthreads();
        } else {
          group_barrier(group);
        }
        products(ps);
      }
      if constexpr (Fix::kFixed) {
        int c[5] = {0, 0, 0, 0, 0};
        bool sure[5] = {true, true, true, true, true};
        sure[0] = nearest_column<kC0>(s0a, n0.a, far0.x, c[0]);
        sure[1] = nearest_column<kC0>(s0b, n0.b, far0.y, c[1]);
        if constexpr (Fix::C1 > 0) {
          sure[2] = nearest_column<kC1>(s1a, n0.a, far1.x, c[2]);
          sure[3] = nearest_column<kC1>(s1b, n0.b, far1.y, c[3]);
        }
        if constexpr (Fix::C2 > 0) sure[4] = nearest_column<kC2>(s2, n0.ab, far2, c[4]);
        if (__any_sync(0xffffffffu, have && (lost || !(sure[0] && sure[1] && sure[2] && sure[3] && sure[4])))) {
          const float far[5] = {far0.x, far0.y, far1.x, far1.y, far2};
          int firsts = 0;
#pragma unroll
          for (int i = 0; i < 5; ++i) {
            const int s = i == 4 ? Fix::kSlots - 1 : i >> 1;
            if ((i >= 2 && i < 4 && Fix::C1 == 0) || (i == 4 && Fix::C2 == 0)) continue;
            // what the first slot's searches found of zeros holds for the others, if their centroids are finite
            const bool first = i >= 2 && far[i] > 0.f && (i == 4 ? firsts == 3 : (firsts >> (i & 1) & 1) != 0);
            if (first) c[i] = 0;
            const unsigned open = __ballot_sync(0xffffffffu, have && (lost || !sure[i]) && !first);
            if (open) {
              const int found = i == 4 ? settle<32>(a, head, s, slice, row, open, c[i]) : settle<16>(a, head, s, 2 * slice + (i & 1), row, open, c[i]);
              c[i] = found & 255;
              if (i < 2) firsts |= (found >> 8 & 1) << i;
            }
          }
        }
        const uint32_t codes[3] = {(uint32_t)(c[0] | (c[1] << 8)), (uint32_t)(c[2] | (c[3] << 8)), (uint32_t)c[4]};
        if (per == 1 || slice != slice0) {  // the group's slices of a row side by side
          if (have) {
            const int64_t at = (int64_t)head * a.rows + row;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              if ((i == 1 && Fix::C1 == 0) || (i == 2 && Fix::C2 == 0)) continue;
              const int s = i == 2 ? Fix::kSlots - 1 : i;
              const int64_t o = i == 2 ? at * (a.dh >> 5) + slice0 : at * (a.dh >> 4) + 2 * slice0;
              const float4 r = per == 1 ? (i == 2 ? make_float4(n0.ab, 0.f, 0.f, 0.f) : make_float4(n0.a, n0.b, 0.f, 0.f))
                                        : (i == 2 ? make_float4(before.ab, n0.ab, 0.f, 0.f) : make_float4(before.a, before.b, n0.a, n0.b));
              store_groups(a.r_out[s] + o, a.th_out[s] + o, per * (i == 2 ? 1 : 2), a.wide, r,
                           per == 1 ? codes[i] : codes_before[i] | codes[i] << (i == 2 ? 8 : 16));
            }
          }
        } else {
          before = n0;
#pragma unroll
          for (int i = 0; i < 3; ++i) codes_before[i] = codes[i];
        }
      }
      if (last_pass) {
        n0 = n1;
        if (next.q < n_q) n1 = convert();
      }
      if (!more) break;
    }
    if (w == 0) waits.leave(wait);
  }
  cp_async_wait<0>();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kSearchGroups * kGroupCols);
  }
}

int validate_tiers(const sphkv_tiers& t, int dh);

}  // namespace sphkv

using namespace sphkv;

struct SearchSmem {
  int codebook_bytes, bytes;
  bool staged;
};
// Staged rows need aligned slices, and room beside a codebook tensor of any C_max (dh 128, four slots a lane: up to 326).
static SearchSmem search_smem(const sphkv_encode_params& p, int tok) {
  const int esize = p.k_dtype == SPHKV_F32 ? 4 : 2;
  const int cb_bytes = p.dh * p.tiers.C_max * 4, row_bytes = 32 * tok * p.dh * 4;
  const bool staged = (reinterpret_cast<uintptr_t>(p.k_src) & 15) == 0 && (p.k_row_stride * esize) % 16 == 0 &&
                      (p.k_head_stride * esize) % 16 == 0 && cb_bytes + row_bytes <= 227 * 1024;
  return {cb_bytes, cb_bytes + (staged ? row_bytes : 0), staged};
}

template <int GS, int TOK>
static int launch_search_parts(const EncodeArgs& a, int resident, cudaStream_t st) {
  static SmemOptIn opt_in[2];
  const sphkv_encode_params& p = a.p;
  const SearchSmem m = search_smem(p, TOK);
  auto kern = m.staged ? search_bundles_kernel<GS, true, TOK> : search_bundles_kernel<GS, false, TOK>;
  if (int rc = ensure_dynamic_smem(opt_in[m.staged], (const void*)kern, m.bytes, "encode search")) return rc;
  EncodeArgs b = a;
  b.search_kbuf = m.codebook_bytes;
  b.search_chunk = std::max(1, std::min(8, p.n_bundles / (resident * 4)));  // >= 4 chunks per CTA, <= 8 bundles each
  const int grid = std::max(1, std::min((p.n_bundles + b.search_chunk - 1) / b.search_chunk, resident));
  (void)launch_overlapped(kern, dim3(grid, 4 / TOK), dim3(kEncThreads), m.bytes, st, b);
  return check_launch("search_bundles_kernel");
}

// Parts that a bundle is cut into while there are few: the search of one alone is half of the launch.  Cut, the CTAs may fill
// four fifths of the chip: blocks of the assembly launch come in early, and where more CTAs leave a few SMs free they pile up
// there (6 and 4 bits, 132 bundles in halves 28.1, without the early launch 22.1).  Quarters of 16-dim groups, two CTAs to
// an SM while the codebooks leave the room, gain up to a full chip.  Encode, dh 128, 148 SMs, us whole / halves / quarters:
//   16 dims, 6 bits      45 bundles 20.1 / 17.0 / 16.9, 73: 20.3 / 18.9 / 17.6, 86: 21.1 / 21.3 / 22.4, 118: 22.7 / 22.1 / 28.0, 130: 22.6 / 28.4 / 30
//   6 and 4 bits         64 bundles 20.2 / 18.8 / 17.7, 96: 20.8 / 18.2 / 19.9, 109: 22.0 / 21.8 / 21.4, 132: 22.2 / 28.1 / 24.4
//   6 bits, one CTA an SM (C_max 196)   32 bundles 20.3 / 16.9 / 15.4, 35: 20.2 / 16.7 / 20.1, 58: 20.3 / 17.7 / 20.5, 68: 20.2 / 24.1 / 22.6
//   32 dims, 3 bits      31 bundles 13.6 / 12.0 / 12.0, 35: 13.4 / 11.9 / 13.2, 58: 13.6 / 12.7 / 11.8, 68: 13.9 / 17.7 / 13.9
static int search_parts(const sphkv_encode_params& p, int gs, int sms) {
  for (int parts = 4; parts >= 2; parts /= 2) {
    const bool two = gs == 16 && 2 * (search_smem(p, 4 / parts).bytes + 1024) <= 228 * 1024;
    const int64_t slots = sms * (two ? 2 : 1), ctas = (int64_t)parts * p.n_bundles;
    if (parts == 4 && two ? ctas <= slots : 5 * ctas <= 4 * slots) return parts;
  }
  return 1;
}

template <int GS>
static int launch_encode(const EncodeArgs& a, bool split, int smem_bytes, cudaStream_t st) {
  if (split) {
    // persistent: as many CTAs as are resident at once, each striding over chunks of bundles
    const int sms = sm_count_current_device(), resident = sms * (GS == 16 ? 2 : 1);
    const int parts = search_parts(a.p, GS, sms);
    return parts == 4   ? launch_search_parts<GS, 1>(a, resident, st)
           : parts == 2 ? launch_search_parts<GS, 2>(a, resident, st)
                        : launch_search_parts<GS, 4>(a, resident, st);
  }
  const int grid = (a.p.n_bundles + a.bundles_per_cta - 1) / a.bundles_per_cta;
  encode_bundle_kernel<GS><<<grid, kEncThreads, smem_bytes, st>>>(a);
  return check_launch("encode_bundle_kernel");
}

// Every page of the bundle list, every tier slot in the same launch: a warp per 16 tokens, so that large pages
// fill the GPU as small ones do.
static int launch_assemble(EncodeArgs& a, bool from_codes, cudaStream_t st) {
  const sphkv_encode_params& p = a.p;
  const int N = p.page_size, GST = p.dh >> 4;
  const int img = ((8 + 4 * GST + N * GST + N * GST * 2) + 15) & ~15;  // 8-bit codes, f16 radii: the largest image
  a.page_smem_bytes = 4 * N + 4 * N * GST + 32 + N * GST + img;
  a.wpp_shift = N == 16 ? 0 : N == 32 ? 1 : N == 64 ? 2 : 3;
  const int at_once = (kEncThreads / 32) >> a.wpp_shift;
  const int smem_bytes = a.page_smem_bytes * at_once;
  static SmemOptIn opt_in[2][2];
  const bool one = a.wpp_shift == 0;
  auto kern = from_codes ? (one ? assemble_pages_kernel<3, true> : assemble_pages_kernel<3, false>)
                         : (one ? assemble_pages_kernel<2, true> : assemble_pages_kernel<2, false>);
  if (int rc = ensure_dynamic_smem(opt_in[from_codes][one], (const void*)kern, smem_bytes, "assemble_pages")) return rc;
  const int64_t items = (int64_t)p.n_bundles * (128 / N);
  const int64_t ctas = (items + at_once - 1) / at_once;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(ctas, (int64_t)sm_count_current_device() * 8));
  (void)launch_overlapped(kern, dim3(grid), dim3(kEncThreads), smem_bytes, st, a);
  return check_launch("assemble_pages_kernel");
}

extern "C" int64_t sphkv_encode_scratch_bytes(int32_t n_pages, int32_t page_size, int32_t dh) {
  if (n_pages <= 0 || page_size <= 0 || dh <= 0) return SPHKV_E_ARG;
  return ((int64_t)n_pages * page_size * (dh / 16) * 5 + 15) / 16 * 16;
}

static int encode_impl(const sphkv_encode_params* pp, void* stream, bool from_codes) {
  SPHKV_REQUIRE(pp != nullptr, SPHKV_E_ARG, "encode: params is NULL");
  const sphkv_encode_params& p = *pp;
  if (p.n_bundles == 0) return 0;
  SPHKV_REQUIRE(p.src_index && p.bundles && p.page_head && p.page_slot && p.ptable && p.k_pages,
                SPHKV_E_ARG, "encode: a required pointer is NULL");
  if (from_codes) {
    SPHKV_REQUIRE(p.code_rows > 0, SPHKV_E_ARG, "pages_from_codes: code_rows=%lld", (long long)p.code_rows);
    for (int s = 0; s < p.tiers.n_slots && s < SPHKV_MAX_TIER_SLOTS; ++s)
      SPHKV_REQUIRE(p.code_r[s] && p.code_theta[s], SPHKV_E_ARG,
                    "pages_from_codes: code cache of tier slot %d is NULL", s);
  } else {
    SPHKV_REQUIRE(p.k_src && p.codebooks, SPHKV_E_ARG, "encode: k_src / codebooks is NULL");
  }
  SPHKV_REQUIRE(p.n_bundles > 0 && p.n_pages > 0, SPHKV_E_ARG, "encode: n_bundles=%d n_pages=%d",
                p.n_bundles, p.n_pages);
  SPHKV_REQUIRE(p.dh == 64 || p.dh == 128, SPHKV_E_ARG, "encode: dh=%d (64 or 128)", p.dh);
  SPHKV_REQUIRE(p.page_size == 16 || p.page_size == 32 || p.page_size == 64 || p.page_size == 128,
                SPHKV_E_ARG, "encode: page_size=%d (16, 32, 64 or 128)", p.page_size);
  SPHKV_REQUIRE(p.k_dtype >= 0 && p.k_dtype <= 2 && p.v_src_dtype >= 0 && p.v_src_dtype <= 2,
                SPHKV_E_DTYPE, "encode: k_dtype=%d v_src_dtype=%d", p.k_dtype, p.v_src_dtype);
  SPHKV_REQUIRE(p.v_pool == nullptr || p.v_pool_dtype == SPHKV_F16 || p.v_pool_dtype == SPHKV_BF16,
                SPHKV_E_DTYPE, "encode: v_pool_dtype=%d", p.v_pool_dtype);
  SPHKV_REQUIRE(p.radius_fmt == SPHKV_RADIUS_I8 || p.radius_fmt == SPHKV_RADIUS_F16, SPHKV_E_ARG,
                "encode: radius_fmt=%d", p.radius_fmt);
  SPHKV_REQUIRE(((uintptr_t)p.k_pages & 3) == 0, SPHKV_E_ALIGN, "encode: k_pages needs 4 B alignment");
  if (int rc = validate_tiers(p.tiers, p.dh)) return rc;
  SPHKV_REQUIRE((from_codes || ((uintptr_t)p.codebooks & 15) == 0) && (p.tiers.g_max & 3) == 0 &&
                    ((uintptr_t)p.v_pool & 15) == 0,
                SPHKV_E_ALIGN, "encode: codebooks / v_pool need 16 B alignment, g_max a multiple of 4");
  // shared memory: codebook of the widest tier + staging + page images
  const int N = p.page_size, TB = 128, ppb = TB / N;
  int smem_bytes = 0;
  for (int s = 0; s < p.tiers.n_slots; ++s) {
    const int G = p.dh / p.tiers.g[s];
    const int img = ((8 + 4 * G + (N * G * p.tiers.bits[s] + 7) / 8 + N * G * 2) + 15) & ~15;
    const int need = p.dh * p.tiers.C_max * 4 + TB * G * 4 + 64 * 4 + 96 + TB * G + 16 + ppb * img;
    smem_bytes = need > smem_bytes ? need : smem_bytes;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  EncodeArgs a;
  a.p = p;
  {  // long runs per CTA amortise the codebook staging, but only once every SM has several CTAs
    int sms = sm_count_current_device();
    if (sms <= 0) sms = 148;
    int bpc = p.n_bundles / (sms * 8);
    a.bundles_per_cta = bpc < 1 ? 1 : (bpc > kMaxBundlesPerCta ? kMaxBundlesPerCta : bpc);
  }
  const int64_t scratch_need = sphkv_encode_scratch_bytes(p.n_pages, p.page_size, p.dh);
  const bool split = p.scratch != nullptr && p.scratch_bytes >= scratch_need &&
                     ((uintptr_t)p.scratch & 15) == 0;
  if (from_codes) return launch_assemble(a, true, st);
  {
    static SmemOptIn opt_in[2];
    const void* kernels[2] = {(const void*)encode_bundle_kernel<16>, (const void*)encode_bundle_kernel<32>};
    for (int i = 0; i < 2; ++i)
      if (int rc = ensure_dynamic_smem(opt_in[i], kernels[i], smem_bytes, "encode")) return rc;
  }
  // One search launch per group size present; each skips the bundles of the other size.
  bool any16 = false, any32 = false;
  for (int s = 0; s < p.tiers.n_slots; ++s) (p.tiers.g[s] == 16 ? any16 : any32) = true;
  if (any16) {
    if (int rc = launch_encode<16>(a, split, smem_bytes, st)) return rc;
  }
  if (any32) {
    if (int rc = launch_encode<32>(a, split, smem_bytes, st)) return rc;
  }
  return split ? launch_assemble(a, false, st) : 0;
}

extern "C" int sphkv_encode_pages(const sphkv_encode_params* p, void* stream) {
  return encode_impl(p, stream, false);
}

extern "C" int sphkv_pages_from_codes(const sphkv_encode_params* p, void* stream) {
  return encode_impl(p, stream, true);
}

static int launch_codes_chains(const CodesArgs& n, int Hkv, cudaStream_t st) {
  ChainArgs a;
  a.k_src = n.k_src; a.codebooks = n.codebooks;
  a.k_row_stride = n.k_row_stride; a.k_head_stride = n.k_head_stride; a.rows = n.rows;
  a.k_dtype = n.k_dtype; a.dh = n.dh; a.tiers = n.tiers;
  int off = 0;
  for (int s = 0; s < SPHKV_MAX_TIER_SLOTS; ++s) {
    a.r_out[s] = n.r_out[s];
    a.th_out[s] = n.th_out[s];
    a.cb_off[s] = off;
    if (s < a.tiers.n_slots) off += a.dh << a.tiers.bits[s];  // G_s * C_s * g_s floats
  }
  // row blocks staged through shared memory when every 32-element slice starts on a 16-byte
  // boundary and the blocks fit beside the codebooks
  const int esz = a.k_dtype == SPHKV_F32 ? 4 : 2;
  const bool aligned = (reinterpret_cast<uintptr_t>(a.k_src) & 15) == 0 && (a.k_row_stride * esz) % 16 == 0 &&
                       (a.k_head_stride * esz) % 16 == 0;
  a.kbuf_off = off * 4;
  const int64_t sms = sm_count_current_device();
  const int row_sets = (kChainThreads / 32) / (a.dh >> 5);  // warps' row sets of a CTA
  auto launch = [&](auto tok) -> int {
    constexpr int TOK = decltype(tok)::value;
    const int kbuf_bytes = (kChainThreads / 32) * 32 * TOK * 128;
    const bool staged = aligned && off * 4 + kbuf_bytes <= 220 * 1024;
    const int smem_bytes = off * 4 + (staged ? kbuf_bytes : 0);
    auto kern = staged ? codes_chains_kernel<true, TOK> : codes_chains_kernel<false, TOK>;
    static SmemOptIn opt_in[2];
    if (int rc = ensure_dynamic_smem(opt_in[staged], (const void*)kern, smem_bytes, "encode_codes")) return rc;
    const int per_cta = row_sets * 32 * TOK;  // rows per CTA and pass
    a.units_per_head = (a.rows + per_cta - 1) / per_cta;
    a.n_units = a.units_per_head * Hkv;
    const dim3 grid((unsigned)std::max<int64_t>(1, std::min(a.n_units, sms)));
    kern<<<grid, kChainThreads, smem_bytes, st>>>(a);
    return 0;
  };
  // Tokens per thread: the fewest microseconds of passes per CTA.  A pass of 4 / 2 / 1 tokens per thread was
  // measured at 24 / 13 / 9 us (three reference tiers; the ratio is what counts): two or one win where four
  // would leave SMs without a unit or the last pass nearly empty.
  auto passes = [&](int tok) {
    const int64_t units = (a.rows + row_sets * 32 * tok - 1) / (row_sets * 32 * tok) * Hkv;
    return (units + sms - 1) / sms;
  };
  const int64_t t4 = passes(4) * 24, t2 = passes(2) * 13, t1 = passes(1) * 9;
  const int rc = t4 <= t2 && t4 <= t1 ? launch(std::integral_constant<int, 4>())
                 : t2 <= t1           ? launch(std::integral_constant<int, 2>())
                                      : launch(std::integral_constant<int, 1>());
  if (rc) return rc;
  return check_launch("codes_chains_kernel");
}

extern "C" int sphkv_encode_codes(const void* k_src, int32_t k_dtype, int64_t k_row_stride,
                                  int64_t k_head_stride, int64_t rows, int32_t Hkv, int32_t dh,
                                  const float* codebooks, const sphkv_tiers* tiers, float* const* r_out,
                                  uint8_t* const* theta_out, void* stream) {
  SPHKV_REQUIRE(k_src && codebooks && tiers && r_out && theta_out, SPHKV_E_ARG, "encode_codes: NULL pointer");
  SPHKV_REQUIRE(rows >= 0 && Hkv > 0 && (dh == 64 || dh == 128) && k_dtype >= 0 && k_dtype <= 2, SPHKV_E_ARG,
                "encode_codes: rows=%lld Hkv=%d dh=%d k_dtype=%d", (long long)rows, Hkv, dh, k_dtype);
  if (int rc = validate_tiers(*tiers, dh)) return rc;
  SPHKV_REQUIRE(((uintptr_t)codebooks & 15) == 0 && (tiers->g_max & 3) == 0, SPHKV_E_ALIGN,
                "encode_codes: codebooks need 16 B alignment, g_max a multiple of 4");
  if (rows == 0) return 0;
  CodesArgs a;
  a.k_src = k_src; a.codebooks = codebooks;
  a.k_row_stride = k_row_stride; a.k_head_stride = k_head_stride; a.rows = rows;
  a.k_dtype = k_dtype; a.dh = dh; a.tiers = *tiers;
  unsigned wanted = 0;
  uintptr_t ends = 0;
  for (int s = 0; s < SPHKV_MAX_TIER_SLOTS; ++s) {
    a.r_out[s] = s < tiers->n_slots ? r_out[s] : nullptr;
    a.th_out[s] = s < tiers->n_slots ? theta_out[s] : nullptr;
    if (s < tiers->n_slots) {
      SPHKV_REQUIRE((a.r_out[s] == nullptr) == (a.th_out[s] == nullptr), SPHKV_E_ARG,
                    "encode_codes: slot %d needs both r_out and theta_out (or neither)", s);
      if (a.r_out[s] != nullptr) {
        wanted |= 1u << s;
        ends |= reinterpret_cast<uintptr_t>(a.r_out[s]) | reinterpret_cast<uintptr_t>(a.th_out[s]) << 2;
      }
      SPHKV_REQUIRE((reinterpret_cast<uintptr_t>(a.r_out[s]) & 7) == 0 && (reinterpret_cast<uintptr_t>(a.th_out[s]) & 1) == 0,
                    SPHKV_E_ARG, "encode_codes: slot %d outputs must be 8-byte (r) and 2-byte (theta) aligned", s);
    }
  }
  SPHKV_REQUIRE(wanted != 0, SPHKV_E_ARG, "encode_codes: no output requested");
  // rows staged through shared memory when every 32-element slice starts on a 16-byte boundary (and, below, where they fit beside
  // the centroids: not with four 64-centroid slots)
  const int esz = k_dtype == SPHKV_F32 ? 4 : 2;
  const bool aligned = (reinterpret_cast<uintptr_t>(k_src) & 15) == 0 && (k_row_stride * esz) % 16 == 0 && (k_head_stride * esz) % 16 == 0;
  // The chains cost 1.2 instructions per centroid and dim; the tensor-core kernel has 5 us of set-up and 45 us for 32768 tokens x 8 heads
  // whatever it searches.  Chains / tensor cores in us at dh 128 by the centroids (of a 32-dim slot, with fewer compares to
  // a dim, 15 of 16 count), 8 heads of 1000, 2048, 4096 and 32768 fp32 tokens:
  //   16: 5 / 9, 6 / 9, 9 / 12, 48 / 50        24: 6 / 11, 8 / 11, 11 / 14, 64 / 64        32: 7.0 / 9.9, 8.8 / 10.3, 12.6 / 13.3, 73 / 55
  //   48: 9.3 / 12.0, 11.8 / 12.2, 17.2 / 16.4, 104 / 71      64: 10.8 / 12.3, 13.7 / 12.3, 20.2 / 16.1, 123 / 66
  //   80: 13.1 / 12.8, 16.8 / 13.4, 24.9 / 16.9, 154 / 64
  // so the lines lie where the chains need more than one round of blocks with four, two or one tokens per thread.  Keys off a 16-byte
  // boundary, 88 centroids: 18.5 / 26.1, 26.2 / 25.6, 43 / 40, 274 / 207.  At dh 64 (half the centroids to lay out) 64 centroids
  // take 9.5 / 8.1 from 64 tokens on, with such keys 13.7 / 12.3.
  int centroids = 0;
  for (int s = 0; s < tiers->n_slots; ++s) centroids += (wanted >> s) & 1u ? (1 << tiers->bits[s]) * (tiers->g[s] == 32 ? 15 : 16) : 0;
  centroids /= 16;
  const auto one_round = [&](int tok) { return (rows + 64 * tok - 1) / (64 * tok) * Hkv <= sm_count_current_device(); };
  const bool chains = dh == 64 ? centroids < 45
                               : centroids < 30 || (centroids < 45 && one_round(4)) || (centroids < 64 && one_round(2)) ||
                                     ((centroids < 80 || !aligned) && one_round(1));
  if (chains) return launch_codes_chains(a, Hkv, reinterpret_cast<cudaStream_t>(stream));
  a.wide = (ends & 15) == 0;
  a.plan = plan_search(*tiers, dh, wanted);
  a.kbuf_off = a.plan.bytes + kCodeTail;
  const int staged_bytes = kSearchThreads / 32 * kCodeStages * kSliceBlock;
  const bool staged = aligned && a.kbuf_off + staged_bytes <= 227 * 1024;
  const int smem_bytes = a.kbuf_off + (staged ? staged_bytes : 0);
  // The reference's tiers (its first two, or all three) have a kernel of their own: 172 us with the chains, 89 us with branches
  // and loops over the slots, 79 us with their sums in registers at once (32768 fp32 tokens x 8 heads, three tiers).
  using Two = FixedTiers<6, 4, 0>;
  using Three = FixedTiers<6, 4, 3>;
  const int which = !staged ? 0 : Three::match(*tiers, wanted) ? 3 : Two::match(*tiers, wanted) ? 2 : 1;
  auto kern = which == 3   ? encode_codes_kernel<true, Three>
              : which == 2 ? encode_codes_kernel<true, Two>
              : which == 1 ? encode_codes_kernel<true, AnyTiers>
                           : encode_codes_kernel<false, AnyTiers>;
  static SmemOptIn opt_in[4];
  if (int rc = ensure_dynamic_smem(opt_in[which], (const void*)kern, smem_bytes, "encode_codes")) return rc;
  a.units_per_head = (rows + 127) / 128;
  a.n_units = a.units_per_head * Hkv;
  const dim3 grid((unsigned)std::max<int64_t>(1, std::min<int64_t>(a.n_units, sm_count_current_device())));
  kern<<<grid, kSearchThreads, smem_bytes, reinterpret_cast<cudaStream_t>(stream)>>>(a);
  return check_launch("encode_codes_kernel");
}
