// Angle-domain decode attention over bit-packed, paged, codebook-quantised keys: host side, RoPE table,
// merge of the split-K partial rows and the exchange between GPUs.  The kernel that reads the pages is in
// splitk.cuh: one persistent CTA per SM walks a range of (KV head, batch row) blocks; three teams of warps
// rebuild keys from page bytes into tensor memory, driver warps fetch (TMA, cp.async) and issue the two
// contractions on the tensor cores.  CTA partials land in scratch and the merge kernel here combines
// them by log-sum-exp.
//
// Numerics restate SphericalKVPipeline._compressed_head_attention_batched
// (spherical_kv_pipeline.py:2136-2177): logit = sum_g r_g * (q_rot_g . c_g) / sqrt(dh)
// with q back-rotated by the key position; rotating the rebuilt key forward instead is the
// same bilinear form.  Page bytes follow pagebuilder.py:8-33 / paging.py:20-31.
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>

#include "splitk.cuh"

namespace sphkv {

constexpr int kMaxUnitsInKernelPlan = 2048;

// ---- RoPE table ------------------------------------------------------------------------
// Row of one position, in the order in which the lanes of the decode kernel consume it (lane_freq): for loop
// index i and lane quad member j, {cos x 4, sin x 4}: 32 bytes per (i, j), so what the four lanes of a
// token read in one step is one 128-byte line.
__global__ void rope_table_kernel(float* __restrict__ table, int max_pos, int dh,
                                  const float* __restrict__ inv_freq) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int half = dh / 2;
  if (idx >= (int64_t)max_pos * half) return;
  const int pos = (int)(idx / half), q = (int)(idx - (int64_t)pos * half);
  const int e = q & 3, j = (q >> 2) & 3, i = q >> 4;
  const int f = lane_freq(dh, i, j, e);
  const float ang = __fmul_rn((float)pos, inv_freq[f]);
  double sn, cs;
  sincos((double)ang, &sn, &cs);
  float* row = table + (int64_t)pos * dh + (i * 4 + j) * 8;
  row[e] = (float)cs;
  row[4 + e] = (float)sn;
}

// ---- plan: exclusive prefix of blocks per unit --------------------------------------
__global__ void plan_kernel(const int32_t* __restrict__ num_blocks, int n_units, int max_blocks,
                            int B, int Hkv, int32_t* __restrict__ pfx) {
  __shared__ int s_part[32];
  __shared__ int s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base = 0; base < n_units; base += blockDim.x) {
    int i = base + threadIdx.x;
    int v = 0;
    if (i < n_units) {
      v = num_blocks[(i % B) * Hkv + i / B];  // traversal order: KV head major, batch row minor
      v = v < 0 ? 0 : (v > max_blocks ? max_blocks : v);
    }
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_part[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = (lane < (int)(blockDim.x >> 5)) ? s_part[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      s_part[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    int carry = s_carry;
    int excl = carry + (warp > 0 ? s_part[warp - 1] : 0) + x - v;
    if (i < n_units) pfx[i] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) pfx[n_units] = s_carry;
}

// grid (unit, importance slices); one thread per (query head, dimension): grp * DH threads.  Bound: memory
// latencies in a row (span -> rows -> output), so everything that can be is loaded at once.  A step of eight
// units, dh 64: 5.3 -> 3.7 us; with the importance update of three rows at 128-token pages 12.3 -> 4.9 us.
template <int DH>
__global__ void __launch_bounds__(8 * DH) merge_rows_kernel(const DecodeArgs a) {
  constexpr int kChunk = 32;   // partial rows combined per pass (general path)
  constexpr int kBatch = 16;   // rows' loads in flight at a time
  const sphkv_decode_params& p = a.p;
  const int u = blockIdx.x;  // traversal index: hkv * B + b
  const int hkv = u / p.B, b = u - hkv * p.B;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = threadIdx.x / DH, d = threadIdx.x % DH;  // this thread's query head (warp-uniform) and dimension
  __shared__ float s_M[8], s_L[8];
  __shared__ union {
    float w[8][kChunk];
    struct { float m[SPHKV_MAX_XCHG_RANKS][8], l[SPHKV_MAX_XCHG_RANKS][8]; } rank;  // exchange: the ranks' rows
  } s_u;
  auto& s_w = s_u.w;
  // launched like the decode kernel: its blocks wait here for it to end, and let the next step's in early
  griddep_wait();
  griddep_launch();
  const int unit = b * p.Hkv + hkv;
  // the CTAs that wrote a partial row of this unit, as the decode kernel's CTAs left them
  int c_lo = 0, nrows = 0;
  const int nb_unit = min(p.num_blocks[unit], p.max_blocks);
  const uint32_t span = a.spans[u];
  if (nb_unit > 0) {
    c_lo = (int)(span & 0xFFFFu);
    nrows = (int)(span >> 16);
  }
  const int64_t row_stride = 8 * (DH + 2);
  const float* rows_n = a.rows + ((int64_t)(c_lo + u) * 8 + n) * (DH + 2);  // row 0 of this thread's head
  float o_acc = 0.f;
  const bool few_rows = nrows <= 32;
  if (few_rows) {
    // At most one row per lane (the usual case: units >= CTAs / 32).  Lane c fetches row c's (max, sum)
    // while the accumulator loads of the first rows are already in flight, the warp reduces, and every
    // lane then folds the rows of its dimension with the weights passed around by shuffles -- one memory
    // latency instead of the four of the general path below, and the same arithmetic in the same order.
    const bool mine = lane < nrows;
    const float mr = mine ? rows_n[lane * row_stride] : -INFINITY;
    const float lr = mine ? rows_n[lane * row_stride + 1] : 0.f;
    float w = 0.f;
    for (int ci = 0; ci < max(nrows, 1); ci += kBatch) {
      float v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) v[k] = ci + k < nrows ? rows_n[(ci + k) * row_stride + 2 + d] : 0.f;
      if (ci == 0) {
        float M = mr;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        w = (mine && M != -INFINITY) ? exp2f(mr - M) : 0.f;
        float L = lr * w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        if (d == 0) { s_M[n] = M; s_L[n] = L; }
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const float wk = __shfl_sync(0xffffffffu, w, (ci + k) & 31);
        o_acc += (ci + k < nrows && wk != 0.f) ? wk * v[k] : 0.f;
      }
    }
  } else if (warp < a.grp) {
    // pass 1: warp h -> global max and sum of head h
    const float* rows_h = a.rows + ((int64_t)(c_lo + u) * 8 + warp) * (DH + 2);
    float M = -INFINITY;
    for (int i = lane; i < nrows; i += 32) M = fmaxf(M, rows_h[i * row_stride]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float L = 0.f;
    if (M != -INFINITY)
      for (int i = lane; i < nrows; i += 32) {
        const float mw = rows_h[i * row_stride];
        if (mw != -INFINITY) L += rows_h[i * row_stride + 1] * exp2f(mw - M);
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    if (lane == 0) { s_M[warp] = M; s_L[warp] = L; }
  }
  __syncthreads();
  // page-importance EMA (_omega_ema_eager, spherical_kv_pipeline.py:952-987) from the per-tile
  // (max, sum) the split-K kernel left in page_ml: per query head the block weights
  // exp(max(m - m_max, -60)) * l are normalised over the blocks, averaged over the heads of
  // this KV head and blended into omega.  m_max is the head's global maximum found above, and
  // the normaliser (the sum of the weights over all blocks) is the head's global sum: both
  // are sums of the same exp(logit - m_max) terms, so no second pass over the blocks is needed
  // (the -60 clamp changes terms below e^-60 of the largest one).
  if (p.omega != nullptr) {
    // A thread takes one (block, query head), gp = grp rounded up to a power of two of them side by side, and
    // loads all (at most eight) tiles of the block at once.  The blocks are spread over gridDim.y CTAs of this
    // unit; each repeats the cheap pass 1.
    const int tpp = p.page_size >> 4;
    const int gp_shift = a.grp <= 1 ? 0 : 32 - __clz(a.grp - 1), gp = 1 << gp_shift;
    const int32_t* bt = p.block_table + (int64_t)unit * p.max_blocks;
    const float one_minus = (1.0f - p.ema_beta) / (float)a.grp;
    const int h = threadIdx.x & (gp - 1);
    const int per_cta = blockDim.x >> gp_shift;
    // (max, sum) pairs as two 4-byte loads: page_ml is the caller's and need not start on 8 bytes
    const float* ml = p.page_ml + ((int64_t)b * p.Hq + (int64_t)hkv * a.grp + min(h, a.grp - 1)) * p.max_blocks * tpp * 2;
    for (int blk0 = blockIdx.y * per_cta; blk0 < p.max_blocks; blk0 += gridDim.y * per_cta) {
      const int blk = blk0 + (threadIdx.x >> gp_shift);
      const bool in = (int)(threadIdx.x >> gp_shift) < per_cta && blk < p.max_blocks;
      float mass = 0.f;
      if (in && h < a.grp && blk < nb_unit && bt[blk] >= 0) {
        float2 t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float* pair = ml + 2 * ((int64_t)blk * tpp + i);
          t[i] = i < tpp ? make_float2(pair[0], pair[1]) : make_float2(-INFINITY, 0.f);
        }
        float m = -INFINITY, l = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (t[i].y > 0.f) m = fmaxf(m, t[i].x);
        if (m != -INFINITY) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (t[i].y > 0.f) l += t[i].y * __expf(t[i].x - m);
          mass = __expf(fmaxf(m - s_M[h] * kLn2, -60.f)) * l / fmaxf(s_L[h], 1e-12f);
        }
      }
      for (int o = 1; o < gp; o <<= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
      if (in && h == 0) {
        float* dst = p.omega + (int64_t)unit * p.max_blocks + blk;
        *dst = *dst * p.ema_beta + mass * one_minus;
      }
    }
  }
  if (blockIdx.y != 0) return;  // only the first CTA of a unit writes the attention output
  // pass 2 of the general path: weights per chunk of rows, then threads over (head, dim)
  for (int c0 = 0; c0 < (few_rows ? 0 : nrows); c0 += kChunk) {
    const int nc = min(kChunk, nrows - c0);
    for (int i = threadIdx.x; i < a.grp * nc; i += blockDim.x) {
      const int h = i / nc, ci = i - h * nc;
      const float mw = a.rows[((int64_t)(c_lo + c0 + ci + u) * 8 + h) * (DH + 2)];
      s_w[h][ci] = (mw == -INFINITY || s_M[h] == -INFINITY) ? 0.f : exp2f(mw - s_M[h]);
    }
    __syncthreads();
    const float* col = rows_n + c0 * row_stride + 2 + d;
    for (int ci = 0; ci < nc; ci += kBatch) {
      float v[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) v[k] = ci + k < nc ? col[(ci + k) * row_stride] : 0.f;
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const float w = ci + k < nc ? s_w[n][ci + k] : 0.f;
        o_acc += w != 0.f ? w * v[k] : 0.f;
      }
    }
    __syncthreads();
  }
  const int64_t hq = (int64_t)b * p.Hq + (int64_t)hkv * a.grp + n;
  {
    const float M = s_M[n], l = s_L[n];
    if (p.out_partial != nullptr) {
      float* dst = p.out_partial + hq * (DH + 2);
      if (d == 0) {
        dst[0] = M * kLn2;
        dst[1] = l;
      }
      dst[2 + d] = o_acc;
    }
    if (p.out != nullptr && p.xchg_world <= 1)
      store_from_float(p.out, p.out_dtype, hq * DH + d, l > 0.f ? o_acc / l : 0.f);
  }
  if (p.xchg_world <= 1) return;

  // ---- split-KV exchange: this rank's rows of the unit go to every rank, then the unit is
  //      combined over the ranks here.  Every 64-bit word a rank stores carries the step number
  //      beside the value ((seq << 32) | f32 bits, one single-copy-atomic store), so a word
  //      validates itself: no fence, no separate flag, one NVLink crossing per value.  Peer
  //      memory is touched by plain stores only; the words a rank reads are in its own memory.
  __shared__ int s_seq, s_ok;
  auto& s_rm = s_u.rank.m;
  auto& s_rl = s_u.rank.l;
  const int64_t n_rows = (int64_t)p.B * p.Hq;
  if (threadIdx.x == 0) {
    s_seq = p.xchg_seq[unit] + 1;
    s_ok = 1;
  }
  __syncthreads();
  const uint32_t seq = (uint32_t)s_seq;
  const int64_t slot_base = (int64_t)(seq & 1) * p.xchg_world * n_rows;  // rows; the two slots alternate by step
  auto put = [&](unsigned long long* dst, float v) {
    const unsigned long long w = ((unsigned long long)seq << 32) | (unsigned long long)__float_as_uint(v);
    asm volatile("st.relaxed.sys.global.b64 [%0], %1;" ::"l"(dst), "l"(w) : "memory");
  };
  {
    const int64_t off = (slot_base + (int64_t)p.xchg_rank * n_rows + hq) * (DH + 2);
    for (int peer = 0; peer < p.xchg_world; ++peer) {
      unsigned long long* dst = p.xchg_recv[peer] + off;
      if (d == 0) {
        put(dst, s_M[n] * kLn2);
        put(dst + 1, s_L[n]);
      }
      put(dst + 2 + d, o_acc);
    }
  }
  // Bounded wait, word by word: a word of this step's slot is in when it carries exactly this
  // step's number (a later step of a peer goes to the other slot; a peer cannot be two steps
  // ahead because it needs this rank's next step to finish its own).  The wait also runs when
  // no output is wanted: it is what keeps the ranks within one step of each other.
  const unsigned long long* mine = p.xchg_recv[p.xchg_rank] + slot_base * (DH + 2);
  const long long limit = p.xchg_timeout_cycles > 0 ? p.xchg_timeout_cycles : 2000000000LL;
  const long long t0 = clock64();
  auto get = [&](const unsigned long long* src) -> float {
    for (;;) {
      unsigned long long w;
      asm volatile("ld.relaxed.sys.global.b64 %0, [%1];" : "=l"(w) : "l"(src) : "memory");
      if ((uint32_t)(w >> 32) == seq) return __uint_as_float((uint32_t)w);
      if (clock64() - t0 > limit) {
        s_ok = 0;  // every thread that gives up writes the same value
        return 0.f;
      }
    }
  };
  for (int i = threadIdx.x; i < p.xchg_world * a.grp; i += blockDim.x) {
    const int rr = i / a.grp, h = i - rr * a.grp;
    const unsigned long long* pr = mine + ((int64_t)rr * n_rows + (int64_t)b * p.Hq + (int64_t)hkv * a.grp + h) * (DH + 2);
    const float pm = get(pr), pl = get(pr + 1);
    s_rm[rr][h] = pl > 0.f ? pm : -INFINITY;
    s_rl[rr][h] = pl;
  }
  __syncthreads();
  float res;
  {
    float M = -INFINITY;
    for (int rr = 0; rr < p.xchg_world; ++rr) M = fmaxf(M, s_rm[rr][n]);
    float l = 0.f, o = 0.f;
    for (int rr = 0; rr < p.xchg_world; ++rr) {
      const float v = get(mine + ((int64_t)rr * n_rows + hq) * (DH + 2) + 2 + d);  // every word is awaited
      if (M == -INFINITY || s_rm[rr][n] == -INFINITY) continue;
      const float w = __expf(s_rm[rr][n] - M);
      l += s_rl[rr][n] * w;
      o += v * w;
    }
    res = l > 0.f ? o / l : 0.f;
  }
  __syncthreads();  // every wait has ended, one way or the other
  if (threadIdx.x == 0) p.xchg_seq[unit] = (int32_t)seq;
  const bool ok = s_ok != 0;
  if (!ok && threadIdx.x == 0 && p.status) atomicOr(p.status, SPHKV_ST_TIMEOUT);  // a rank never published this step
  if (p.out == nullptr) return;
  store_from_float(p.out, p.out_dtype, hq * DH + d, ok ? res : 0.f);  // defined output either way
}

// ---- merge of R partial sets (cross-GPU split-KV) ----------------------------------------
__global__ void merge_partials_kernel(const float* __restrict__ parts, int R, int n_rows, int dh,
                                      void* __restrict__ out, int out_dtype) {
  const int row = blockIdx.x;
  const int64_t stride = (int64_t)n_rows * (dh + 2);
  float M = -INFINITY;
  for (int rr = 0; rr < R; ++rr) {
    const float* pr = parts + rr * stride + (int64_t)row * (dh + 2);
    if (pr[1] > 0.f) M = fmaxf(M, pr[0]);
  }
  for (int d = threadIdx.x; d < dh; d += blockDim.x) {
    float l = 0.f, o = 0.f;
    if (M != -INFINITY) {
      for (int rr = 0; rr < R; ++rr) {
        const float* pr = parts + rr * stride + (int64_t)row * (dh + 2);
        if (!(pr[1] > 0.f)) continue;
        const float w = __expf(pr[0] - M);
        l += pr[1] * w;
        o += pr[2 + d] * w;
      }
    }
    store_from_float(out, out_dtype, (int64_t)row * dh + d, l > 0.f ? o / l : 0.f);
  }
}

// ---- host side --------------------------------------------------------------------------------
static int64_t align_up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

// Shared-memory layout of the codebooks: a g = 16 slot may be stored twice (row pitch 128
// bytes, second copy for odd token rows) when the policy asks for it and the space is there.
static int smem_cb_layout(const sphkv_tiers& t, int dh, int budget_bytes, int* offs, int* dup) {
  int plain = 0;
  for (int s = 0; s < t.n_slots; ++s) plain += dh * (1 << t.bits[s]) * 4 + kCbShift;
  int extra_left = budget_bytes - plain;
  int off = 0;
  for (int s = 0; s < t.n_slots; ++s) {
    const int bytes = dh * (1 << t.bits[s]) * 4 + kCbShift;
    const bool want = t.g[s] == 16;
    dup[s] = (want && bytes <= extra_left) ? 1 : 0;
    if (dup[s]) extra_left -= bytes;
    offs[s] = off;
    off += bytes * (dup[s] ? 2 : 1);
  }
  return off;
}

// all that a block can have: the decode kernel's 512 threads launch with every register of an SM, so its blocks never
// share one with the merge blocks of the step before, and overlap with them on the SMs that have none
constexpr int kSmemMax = 227 * 1024;

// Shared memory of a decode: as many teams as fit beside every codebook and the block prefix (0: not one), then the copies of
// codebooks that still do.  Returns the bytes.
static int plan_smem(const sphkv_tiers& t, int dh, int n_units, int& teams, int* offs, int* dup, int& cb_bytes) {
  const int pfx_bytes = n_units <= kMaxUnitsInKernelPlan ? (n_units + 1) * 4 : 0;
  int bytes = 0;
  for (teams = kTeams; teams >= 1; --teams) {
    const int fixed_bytes = smem_fixed_bytes(dh, teams) + pfx_bytes;
    cb_bytes = smem_cb_layout(t, dh, kSmemMax - fixed_bytes, offs, dup);
    bytes = fixed_bytes + cb_bytes;
    if (bytes <= kSmemMax) break;
  }
  return bytes;
}

int validate_tiers(const sphkv_tiers& t, int dh) {
  SPHKV_REQUIRE(t.n_slots >= 1 && t.n_slots <= SPHKV_MAX_TIER_SLOTS, SPHKV_E_ARG,
                "tiers.n_slots=%d outside 1..%d", t.n_slots, SPHKV_MAX_TIER_SLOTS);
  for (int s = 0; s < t.n_slots; ++s) {
    SPHKV_REQUIRE(t.g[s] == 16 || t.g[s] == 32, SPHKV_E_ARG, "tier slot %d: g=%d (16 or 32)", s,
                  t.g[s]);
    SPHKV_REQUIRE(t.bits[s] >= 1 && t.bits[s] <= 6, SPHKV_E_ARG, "tier slot %d: bits=%d (1..6)", s,
                  t.bits[s]);
    SPHKV_REQUIRE(dh % (2 * t.g[s]) == 0, SPHKV_E_ARG, "tier slot %d: dh=%d not a multiple of 2g",
                  s, dh);
    SPHKV_REQUIRE(dh / t.g[s] <= t.G_max && (1 << t.bits[s]) <= t.C_max && t.g[s] <= t.g_max,
                  SPHKV_E_ARG, "tier slot %d exceeds codebook tensor (G_max=%d C_max=%d g_max=%d)",
                  s, t.G_max, t.C_max, t.g_max);
  }
  return 0;
}

// ---- tensor map of the V pool ------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
    tried = true;
  }
  return fn;
}

// V pool viewed as a 3-D tensor [dh / 64][n_pages * page_size rows][64] of 16-bit elements; a box is all the
// 64-element slices (128 bytes, the widest row the 128-byte swizzle takes) of 16 rows, so a tile is one
// copy.  Encoding is host arithmetic only (no device memory, no driver state).
static int make_v_map(CUtensorMap* map, const sphkv_decode_params& p) {
  EncodeTiledFn fn = encode_tiled_fn();
  SPHKV_REQUIRE(fn != nullptr, SPHKV_E_ARG, "decode: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[3] = {64, (cuuint64_t)p.n_pages * (cuuint64_t)p.page_size, (cuuint64_t)p.dh / 64};
  const cuuint64_t strides[2] = {(cuuint64_t)p.dh * 2, 128};
  const cuuint32_t box[3] = {64, 16, (cuuint32_t)p.dh / 64};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult rc = fn(map, p.v_dtype == SPHKV_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                         3, const_cast<void*>(p.v_pool), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  SPHKV_REQUIRE(rc == CUDA_SUCCESS, SPHKV_E_ARG, "decode: cuTensorMapEncodeTiled failed (%d) for the V pool", (int)rc);
  return 0;
}

template <int DH, typename VT, bool ROT, int MODE, bool PACK>
static int launch_decode_t(const DecodeArgs& a, int smem_bytes, cudaStream_t st) {
  static SmemOptIn opt_in;
  auto kern = decode_splitk_kernel<DH, VT, ROT, MODE, PACK>;
  if (int rc = ensure_dynamic_smem(opt_in, (const void*)kern, smem_bytes, "decode")) return rc;
  (void)launch_overlapped(kern, dim3(a.n_ctas), dim3(kDecodeThreads), smem_bytes, st, a);  // check_launch reports
  return check_launch("decode_splitk_kernel");
}

template <int DH, typename VT, bool ROT>
static int launch_decode_r(const DecodeArgs& a, int smem_bytes, cudaStream_t st) {
  const bool extra = a.p.logits_out != nullptr || a.p.page_ml != nullptr;
  const bool pack = a.grp <= 4;
  const bool fast = a.p.page_size == 16 && a.p.radius_fmt == SPHKV_RADIUS_I8;
  if (extra && fast)
    return pack ? launch_decode_t<DH, VT, ROT, 2, true>(a, smem_bytes, st)
                : launch_decode_t<DH, VT, ROT, 2, false>(a, smem_bytes, st);
  if (extra)
    return pack ? launch_decode_t<DH, VT, ROT, 3, true>(a, smem_bytes, st)
                : launch_decode_t<DH, VT, ROT, 3, false>(a, smem_bytes, st);
  if (fast)
    return pack ? launch_decode_t<DH, VT, ROT, 0, true>(a, smem_bytes, st)
                : launch_decode_t<DH, VT, ROT, 0, false>(a, smem_bytes, st);
  return pack ? launch_decode_t<DH, VT, ROT, 1, true>(a, smem_bytes, st)
              : launch_decode_t<DH, VT, ROT, 1, false>(a, smem_bytes, st);
}

template <int DH, typename VT>
static int launch_decode(const DecodeArgs& a, int smem_bytes, cudaStream_t st) {
  return a.p.rope_table != nullptr ? launch_decode_r<DH, VT, true>(a, smem_bytes, st)
                                   : launch_decode_r<DH, VT, false>(a, smem_bytes, st);
}

}  // namespace sphkv

using namespace sphkv;

extern "C" int sphkv_rope_table_build(float* table, int32_t max_pos, int32_t dh,
                                      const float* inv_freq, void* stream) {
  SPHKV_REQUIRE(table && inv_freq, SPHKV_E_ARG, "rope_table: NULL pointer");
  SPHKV_REQUIRE(max_pos > 0 && (dh == 64 || dh == 128), SPHKV_E_ARG, "rope_table: max_pos=%d dh=%d",
                max_pos, dh);
  SPHKV_REQUIRE(((uintptr_t)table & 31) == 0, SPHKV_E_ALIGN, "rope_table: table needs 32-byte alignment");
  const int64_t n = (int64_t)max_pos * (dh / 2);
  rope_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      table, max_pos, dh, inv_freq);
  return check_launch("rope_table_kernel");
}

// Block prefix per unit and the units' spans of CTAs.  One array serves both when the decode kernel derives the
// prefix itself (it keeps it in shared memory).
static int64_t prefix_bytes(int64_t n_units) {
  return align_up((n_units + 1) * 4, 256) * (n_units <= kMaxUnitsInKernelPlan ? 1 : 2);
}

static int resolve_ctas(int n_ctas) { return n_ctas > 0 ? n_ctas : sm_count_current_device(); }

extern "C" int64_t sphkv_decode_scratch_bytes(int32_t B, int32_t Hkv, int32_t dh, int32_t n_ctas) {
  n_ctas = resolve_ctas(n_ctas);
  if (n_ctas <= 0 || B <= 0 || Hkv <= 0 || dh <= 0) return SPHKV_E_ARG;
  const int64_t n_units = (int64_t)B * Hkv;
  return prefix_bytes(n_units) + (int64_t)(n_ctas + n_units) * 8 * (dh + 2) * 4;
}

extern "C" int sphkv_decode_smem(const sphkv_tiers* tiers, int32_t dh, int32_t n_units, int32_t* teams, int32_t* copies) {
  SPHKV_REQUIRE(tiers && teams && copies, SPHKV_E_ARG, "decode_smem: NULL pointer");
  SPHKV_REQUIRE((dh == 64 || dh == 128) && n_units > 0, SPHKV_E_ARG, "decode_smem: dh=%d units=%d", dh, n_units);
  if (int rc = validate_tiers(*tiers, dh)) return rc;
  int offs[SPHKV_MAX_TIER_SLOTS], dup[SPHKV_MAX_TIER_SLOTS], cb_bytes = 0, n = 0;
  const int bytes = plan_smem(*tiers, dh, n_units, n, offs, dup, cb_bytes);
  *teams = n;
  for (int s = 0; s < tiers->n_slots; ++s) copies[s] = 1 + dup[s];
  return bytes;
}

extern "C" int sphkv_decode_paged(const sphkv_decode_params* pp, void* stream) {
  SPHKV_REQUIRE(pp != nullptr, SPHKV_E_ARG, "decode: params is NULL");
  const sphkv_decode_params& p = *pp;
  SPHKV_REQUIRE(p.q && p.k_pages && p.ptable && p.v_pool && p.block_table && p.bits_table &&
                    p.num_blocks && p.codebooks && p.scratch,
                SPHKV_E_ARG, "decode: a required pointer is NULL");
  SPHKV_REQUIRE(p.out || p.out_partial, SPHKV_E_ARG, "decode: out and out_partial both NULL");
  SPHKV_REQUIRE(p.rope_table == nullptr || p.positions != nullptr, SPHKV_E_ARG,
                "decode: rope_table given without positions");
  SPHKV_REQUIRE(p.rope_table == nullptr || p.max_pos > 0, SPHKV_E_ARG,
                "decode: rope_table given with max_pos=%d (rows of the table)", p.max_pos);
  SPHKV_REQUIRE(p.omega == nullptr || p.page_ml != nullptr, SPHKV_E_ARG,
                "decode: omega needs page_ml (the per-tile statistics it is computed from)");
  SPHKV_REQUIRE(p.dh == 64 || p.dh == 128, SPHKV_E_ARG, "decode: dh=%d (64 or 128)", p.dh);
  SPHKV_REQUIRE(p.B > 0 && p.Hkv > 0 && p.Hq > 0 && p.Hq % p.Hkv == 0, SPHKV_E_ARG,
                "decode: B=%d Hq=%d Hkv=%d", p.B, p.Hq, p.Hkv);
  const int grp = p.Hq / p.Hkv;
  SPHKV_REQUIRE(grp <= SPHKV_MAX_GQA, SPHKV_E_LIMIT, "decode: %d query heads per KV head (max %d)",
                grp, SPHKV_MAX_GQA);
  SPHKV_REQUIRE(p.page_size == 16 || p.page_size == 32 || p.page_size == 64 || p.page_size == 128,
                SPHKV_E_ARG, "decode: page_size=%d (16, 32, 64 or 128)", p.page_size);
  SPHKV_REQUIRE(p.max_blocks > 0 && p.n_pages > 0, SPHKV_E_ARG, "decode: max_blocks=%d n_pages=%d",
                p.max_blocks, p.n_pages);
  SPHKV_REQUIRE(p.v_dtype == SPHKV_F16 || p.v_dtype == SPHKV_BF16, SPHKV_E_DTYPE,
                "decode: v_dtype=%d", p.v_dtype);
  SPHKV_REQUIRE(p.q_dtype >= 0 && p.q_dtype <= 2 && p.out_dtype >= 0 && p.out_dtype <= 2,
                SPHKV_E_DTYPE, "decode: q_dtype=%d out_dtype=%d", p.q_dtype, p.out_dtype);
  SPHKV_REQUIRE(p.radius_fmt == SPHKV_RADIUS_I8 || p.radius_fmt == SPHKV_RADIUS_F16, SPHKV_E_ARG,
                "decode: radius_fmt=%d", p.radius_fmt);
  SPHKV_REQUIRE(((uintptr_t)p.v_pool & 15) == 0 && ((uintptr_t)p.k_pages & 3) == 0 &&
                    ((uintptr_t)p.codebooks & 15) == 0 && (p.tiers.g_max & 3) == 0 &&
                    (p.rope_table == nullptr || ((uintptr_t)p.rope_table & 31) == 0) &&
                    ((uintptr_t)p.scratch & 255) == 0,
                SPHKV_E_ALIGN, "decode: v_pool/codebooks need 16 B, rope_table 32 B, k_pages 4 B, scratch 256 B");
  if (int rc = validate_tiers(p.tiers, p.dh)) return rc;
  if (p.xchg_world > 1) {
    SPHKV_REQUIRE(p.xchg_world <= SPHKV_MAX_XCHG_RANKS, SPHKV_E_LIMIT, "decode: xchg_world=%d (max %d)",
                  p.xchg_world, SPHKV_MAX_XCHG_RANKS);
    SPHKV_REQUIRE(p.xchg_rank >= 0 && p.xchg_rank < p.xchg_world, SPHKV_E_ARG, "decode: xchg_rank=%d of %d",
                  p.xchg_rank, p.xchg_world);
    SPHKV_REQUIRE(p.xchg_recv && p.xchg_seq, SPHKV_E_ARG, "decode: the exchange needs xchg_recv and xchg_seq");
    SPHKV_REQUIRE(p.omega == nullptr, SPHKV_E_ARG,
                  "decode: the page-importance update is per rank; run it without the exchange");
  }

  DecodeArgs a;
  a.p = p;
  a.n_ctas = resolve_ctas(p.n_ctas);
  SPHKV_REQUIRE(a.n_ctas > 0, SPHKV_E_ARG, "decode: cannot resolve CTA count");
  a.n_units = p.B * p.Hkv;
  a.grp = grp;
  const int64_t need = sphkv_decode_scratch_bytes(p.B, p.Hkv, p.dh, a.n_ctas);
  SPHKV_REQUIRE(p.scratch_bytes >= need, SPHKV_E_SCRATCH, "decode: scratch %lld B < %lld B",
                (long long)p.scratch_bytes, (long long)need);
  a.pfx = reinterpret_cast<int32_t*>(p.scratch);
  a.rows = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.scratch) + prefix_bytes(a.n_units));
  a.spans = reinterpret_cast<uint32_t*>(p.scratch);
  if (a.n_units > kMaxUnitsInKernelPlan) a.spans += align_up((int64_t)(a.n_units + 1) * 4, 256) / 4;
  a.n_ctas = min(a.n_ctas, 0xFFFF);  // a span packs two CTA counts into a word
  a.wide = ((reinterpret_cast<uintptr_t>(p.k_pages) | reinterpret_cast<uintptr_t>(p.positions)) & 15) == 0;
  a.plan_in_kernel = a.n_units <= kMaxUnitsInKernelPlan ? 1 : 0;
  const int smem_bytes = plan_smem(p.tiers, p.dh, a.n_units, a.teams, a.cb_smem_off, a.cb_dup, a.cb_smem_bytes);
  SPHKV_REQUIRE(a.teams >= 1, SPHKV_E_LIMIT,
                "decode: codebooks need %d B of shared memory (limit %d)", smem_bytes, kSmemMax);
  if (int rc = make_v_map(&a.v_map, p)) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);

  if (!a.plan_in_kernel) {
    plan_kernel<<<1, 1024, 0, st>>>(p.num_blocks, a.n_units, p.max_blocks, p.B, p.Hkv, a.pfx);
    if (int rc = check_launch("plan_kernel")) return rc;
  }
  int rc;
  if (p.dh == 128)
    rc = p.v_dtype == SPHKV_F16 ? launch_decode<128, __half>(a, smem_bytes, st)
                                : launch_decode<128, __nv_bfloat16>(a, smem_bytes, st);
  else
    rc = p.v_dtype == SPHKV_F16 ? launch_decode<64, __half>(a, smem_bytes, st)
                                : launch_decode<64, __nv_bfloat16>(a, smem_bytes, st);
  if (rc) return rc;
  // with an importance update, extra CTAs per unit share the walk over the blocks
  const int merge_threads = grp * p.dh;
  const dim3 mgrid(a.n_units, p.omega ? (unsigned)std::max(1, std::min(16, p.max_blocks * SPHKV_MAX_GQA / merge_threads)) : 1u);
  if (p.dh == 128)
    (void)launch_overlapped(merge_rows_kernel<128>, mgrid, dim3(merge_threads), 0, st, a);
  else
    (void)launch_overlapped(merge_rows_kernel<64>, mgrid, dim3(merge_threads), 0, st, a);
  return check_launch("merge_rows_kernel");
}

extern "C" int sphkv_merge_partials(const float* parts, int32_t R, int32_t n_rows, int32_t dh,
                                    void* out, int32_t out_dtype, void* stream) {
  SPHKV_REQUIRE(parts && out, SPHKV_E_ARG, "merge: NULL pointer");
  SPHKV_REQUIRE(R > 0 && n_rows > 0 && dh > 0, SPHKV_E_ARG, "merge: R=%d n_rows=%d dh=%d", R,
                n_rows, dh);
  SPHKV_REQUIRE(out_dtype >= 0 && out_dtype <= 2, SPHKV_E_DTYPE, "merge: out_dtype=%d", out_dtype);
  merge_partials_kernel<<<n_rows, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      parts, R, n_rows, dh, out, out_dtype);
  return check_launch("merge_partials_kernel");
}
// ---- decode without any caller- or library-side allocation -------------------------------
// Some hosts of this library cannot hand it scratch memory: an inference server that gave
// its whole HBM budget to the KV pools at start-up has nothing left for cudaMalloc to
// return, and a plug-in loaded into such a process has no allocator of its own to ask.  For
// them the split-K scratch of the decode kernels lives in the library image.
//
// Limits (the array is sized for them; every GPU that loads the library carries it until
// the process exits): B * Hkv <= 256 units, at most 160 CTAs, dh <= 128.
#define SPHKV_STATIC_MAX_UNITS 256
#define SPHKV_STATIC_MAX_CTAS 160
#define SPHKV_STATIC_SCRATCH_BYTES \
  (((SPHKV_STATIC_MAX_UNITS + 1) * 4 + 255) / 256 * 256 + \
   (SPHKV_STATIC_MAX_CTAS + SPHKV_STATIC_MAX_UNITS) * 8 * (128 + 2) * 4)
static __device__ __align__(256) unsigned char g_static_scratch[SPHKV_STATIC_SCRATCH_BYTES];

// g_static_scratch names a host-side handle here, not a device address; the address a
// kernel can use comes from cudaGetSymbolAddress, asked once per device with that device
// current.
static void* static_scratch_for_current_device(int* rc_out) {
  static void* cached[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    set_error("decode_static: cudaGetDevice: %s (device %d)", cudaGetErrorString(e), dev);
    *rc_out = e != cudaSuccess ? (int)e : SPHKV_E_LIMIT;
    return nullptr;
  }
  if (cached[dev] == nullptr) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || ptr == nullptr) {
      set_error("decode_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      *rc_out = e != cudaSuccess ? (int)e : SPHKV_E_ARG;
      return nullptr;
    }
    cached[dev] = ptr;
  }
  *rc_out = 0;
  return cached[dev];
}

extern "C" int sphkv_decode_paged_static(const sphkv_decode_params* pp, void* stream) {
  SPHKV_REQUIRE(pp != nullptr, SPHKV_E_ARG, "decode_static: params is NULL");
  SPHKV_REQUIRE(pp->B > 0 && pp->Hkv > 0 && (int64_t)pp->B * pp->Hkv <= SPHKV_STATIC_MAX_UNITS,
                SPHKV_E_LIMIT, "decode_static: B*Hkv=%lld exceeds the built-in scratch (max %d units)",
                (long long)pp->B * pp->Hkv, SPHKV_STATIC_MAX_UNITS);
  SPHKV_REQUIRE(pp->dh > 0 && pp->dh <= 128, SPHKV_E_LIMIT,
                "decode_static: dh=%d exceeds the built-in scratch (max 128)", pp->dh);
  const int n_ctas = resolve_ctas(pp->n_ctas);
  SPHKV_REQUIRE(n_ctas > 0 && n_ctas <= SPHKV_STATIC_MAX_CTAS, SPHKV_E_LIMIT,
                "decode_static: %d CTAs exceed the built-in scratch (max %d); pass n_ctas", n_ctas,
                SPHKV_STATIC_MAX_CTAS);
  int rc = 0;
  void* scratch = static_scratch_for_current_device(&rc);
  if (scratch == nullptr) return rc;
  sphkv_decode_params q = *pp;
  q.n_ctas = n_ctas;
  q.scratch = scratch;
  q.scratch_bytes = SPHKV_STATIC_SCRATCH_BYTES;
  return sphkv_decode_paged(&q, stream);
}
