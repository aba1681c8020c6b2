// Nearest-centroid search on the tensor cores with an exact decision.
//
// What the encoders and k-means promise is the first maximum of fp32 fma chains (k . c over d = 0 .. g-1 from
// 0).  As chains on the fp32 pipe the search costs 16 fmas and three compare / select instructions per
// (16-dim group, centroid).  Here the tensor cores compute every product sum from bf16 pairs (key = hi + lo,
// centroid = hi + lo, four products, fp32 accumulators in tensor memory), a thread looks at its token's row of
// approximate sums at 2.5 instructions per centroid, and the answer is taken only where the largest one leads by
// more than twice what the approximation can be off; where it does not (some 0.1 % of the searches) the
// chains decide.  The result is that of the chains, bit for bit.
//
// Error of an approximate sum, relative to |k| |c| (Cauchy-Schwarz over the dims): a value less its two bf16 parts
// (kPairError), for the key and for the centroid; the chains' own rounding (kChainError); and the tensor core's sums (kSumError).
// Twice all of it is 0.98 kGap; without the product lo * lo, up to 2^-16, it would be 1.6 kGap (k-means leaves it out, with a lead
// of its own).  The tensor core, measured on this part
// (one term 1, fifteen of 2^-18 .. 2^-29): a product's addends are cut off below 2^-25 of the largest, the sum at
// fp32, so a product of 16 addends and the accumulator lose at most 17 x 2^-25 + 2^-23 (seen on random vectors: 2^-21.2 in
// all).  Norms outside 2^-30 .. 2^30 (underflow, overflow, infinities, NaN) are never decided here.
#pragma once
#include "tcgen05.cuh"

namespace sphkv {

constexpr float kGap = 3.f / 65536.f;       // lead over the runner-up, relative to |k| max |c|, that settles a search
constexpr double kPairError = 1. / (1 << 17);                                // half a place of lo, which is at most 2^-8
constexpr double kSumError = 17. / (1 << 25) + 1. / (1 << 23);               // of one product; four for each half of 32 dims
constexpr double kChainError = 32. / (1 << 24);
constexpr double kRestError = 1. / (1 << 23);                                // of norms, t and products of two remainders
static_assert(2 * (2 * kPairError + 8 * kSumError + kChainError + kRestError) < kGap, "the lead covers both sums' errors");
constexpr int kSearchWarps = 4;             // warps of a search group: the 128 lanes (token rows) of tensor memory
constexpr int kSearchGroups = 2;            // search groups of a CTA
constexpr int kSearchThreads = kSearchGroups * kSearchWarps * 32;
constexpr int kGroupCols = 256;             // tensor memory columns of a group ...
constexpr int kSumCols = 192;               // ... of which the sums take up to 192,
constexpr int kKeyCols = 192;               // and two buffers of 32 the key pairs of a 32-dim slice (hi x 16 | lo x 16)

// bf16 pairs of N fp32 values: hi = rounded, lo = rounded rest (off by kPairError at most); word i holds values 2 i and 2 i + 1
template <int N>
__device__ __forceinline__ void split_pairs(const float (&k)[N], uint32_t (&hi)[N / 2], uint32_t (&lo)[N / 2]) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(k[2 * i], k[2 * i + 1]);
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
    const float2 rest = __ffma2_rn(make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u)),
                                   make_float2(-1.f, -1.f), make_float2(k[2 * i], k[2 * i + 1]));
    const __nv_bfloat162 l = __floats2bfloat162_rn(rest.x, rest.y);
    hi[i] = w;
    lo[i] = *reinterpret_cast<const uint32_t*>(&l);
  }
}

__device__ __forceinline__ void tmem_st_x16(uint32_t addr, const uint32_t (&v)[16]) {  // lane = row, 16 columns
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_x8(uint32_t addr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_ld_x32(uint32_t addr, float* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
        "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]),
        "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]),
        "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
      : "r"(addr));
}
// the first C columns at `addr` (lane = row); the caller waits
template <int C>
__device__ __forceinline__ void tmem_ld_row(uint32_t addr, float (&v)[C < 16 ? 16 : C]) {
  if constexpr (C == 64) {
    tmem_ld_x32(addr, v);
    tmem_ld_x32(addr + 32, v + 32);
  } else if constexpr (C == 32) {
    tmem_ld_x32(addr, v);
  } else if constexpr (C == 16) {
    tmem_ld_x16(addr, v);
  } else {
    tmem_ld_x8(addr, v);
  }
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

// One search: column of the largest of v[0 .. C-1], and whether it leads all others by more than kGap |k| max |c|.
// `norm` = |k|, `most` = max |c| (NaN where the centroids' norms are out of range).  The columns above
// t = largest - gap are counted and named in one sum: each adds 1024 + its number, as a saturated multiply-add (1 where
// v > t, else 0: a power of two large enough that the smallest difference from t saturates it) and an fma,
// which the fp32 pipe issues at twice the rate of compare and select.
template <int C>
__device__ __forceinline__ float largest_of(const float (&v)[C < 16 ? 16 : C]) {
  float part[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) part[i] = v[i & (C - 1)];
#pragma unroll
  for (int c = 4; c < C; c += 8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) part[i] = c + 4 + i < C ? max3(part[i], v[c + i], v[(c + 4 + i) & (C - 1)]) : fmaxf(part[i], v[c + i]);
  }
  return fmaxf(max3(part[0], part[1], part[2]), part[3]);
}
struct Lead {
  float gap, t, scale, shift;
  bool fit;  // norms and t in the range where the sums below are exact
};
__device__ __forceinline__ Lead lead_of(float top, float norm, float most, float lead = kGap) {
  Lead l;
  l.gap = lead * norm * most;
  l.t = top - l.gap;
  // 2^36 / 2^exponent(gap): t at least 2^-10 gap away from 0 differs from any other float by 2^-35 gap or more
  l.scale = __uint_as_float((290u - (__float_as_uint(l.gap) >> 23)) << 23);
  l.shift = -l.t * l.scale;
  l.fit = norm >= 9.3132257e-10f && norm <= 1.0737418e9f && most > 0.f && fabsf(l.t) >= l.gap * (1.f / 1024.f);
  return l;
}
template <int C>
__device__ __forceinline__ float count_leaders(const float (&v)[C < 16 ? 16 : C], const Lead& l) {
  float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < C; ++c) sum[c & 3] = __fmaf_rn(__saturatef(__fmaf_rn(v[c], l.scale, l.shift)), (float)(1024 + c), sum[c & 3]);
  return (sum[0] + sum[1]) + (sum[2] + sum[3]);
}
// one leader, or more than one; its number
__device__ __forceinline__ bool one_leader(float all) { return all < 2048.f; }
__device__ __forceinline__ int leader_of(float all) { return __float_as_int(all + 8387584.f) & 1023; }  // 2^23 - 1024: the sum's low bits
template <int C>
__device__ __forceinline__ bool nearest_column(const float (&v)[C < 16 ? 16 : C], float norm, float most, int& code) {
  const Lead l = lead_of(largest_of<C>(v), norm, most);
  const float all = count_leaders<C>(v, l);
  code = leader_of(all);
  return l.fit && one_leader(all);
}

// Norms of a 32-dim slice: its two 16-dim groups and the whole, whose fma chain continues that of the first group
struct SliceNorms {
  float a, b, ab;
};
// fma chains of the norms; the slice's bf16 pairs to tensor memory at `dst` (lane = row), waited for
__device__ __forceinline__ SliceNorms store_slice(const float (&k)[32], uint32_t dst, bool lows) {
  float na = 0.f, nb = 0.f;
#pragma unroll
  for (int d = 0; d < 16; ++d) {
    na = __fmaf_rn(k[d], k[d], na);
    nb = __fmaf_rn(k[16 + d], k[16 + d], nb);
  }
  float nab = na;
#pragma unroll
  for (int d = 16; d < 32; ++d) nab = __fmaf_rn(k[d], k[d], nab);
  uint32_t hi[16], lo[16];
  split_pairs(k, hi, lo);
  tmem_st_x16(dst, hi);
  if (lows) tmem_st_x16(dst + 16, lo);
  const SliceNorms n = {__fsqrt_rn(na), __fsqrt_rn(nb), __fsqrt_rn(nab)};
  tmem_wait_st();
  return n;
}

// Number 0 whatever the chains say: a vector with a NaN has NaN sums only, which never win, and one of zeros has sums of zero, or NaN
// with centroids that are not finite (the first one is looked at).  Padding is such vectors, and whole warps of them.
template <int GS>
__device__ __forceinline__ bool first_wins(const float (&k)[GS], const float* __restrict__ cb) {
  uint32_t largest = 0;
#pragma unroll
  for (int d = 0; d < GS; ++d) largest = max(largest, __float_as_uint(k[d]) & 0x7fffffffu);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < GS / 4; ++i) {
    const float4 x = reinterpret_cast<const float4*>(cb)[i];
    sum = __fmaf_rn(0.f, x.x, __fmaf_rn(0.f, x.y, __fmaf_rn(0.f, x.z, __fmaf_rn(0.f, x.w, sum))));
  }
  return largest == 0 ? sum == 0.f : largest > 0x7f800000u;
}

// sums as integers of the same order; NaN, which never wins, as -inf
__device__ __forceinline__ int ordered(float s) {
  const int i = __float_as_int(s == s ? s + 0.f : -INFINITY);  // (-0 + 0 = 0)
  return i ^ ((i >> 31) & 0x7fffffff);
}
// The chains themselves, for the lanes in `todo` (warp-uniform); k = a lane's group vector, `cb` = the group's centroids, `pitch`
// floats apart.  Lane after lane: the warp's lanes hold centroids in registers and get the vectors by
// shuffles.  More lanes than centroids: every lane walks the centroids for itself.  Returns a lane's code, or `code` where it
// has nothing to do.
template <int GS>
__device__ __forceinline__ int exact_search(const float (&k)[GS], const float* __restrict__ cb, int pitch, int C, unsigned todo, int code) {
  constexpr int kRows = GS >= 32 ? 1 : 2;  // centroids a lane holds
  const int lane = threadIdx.x & 31;
  const bool mine = (todo >> lane) & 1u;
  int best = ordered(-INFINITY);
  if (mine) code = 0;
  if (__popc(todo) > C) {
    if (mine) {
#pragma unroll 1
      for (int c0 = 0; c0 < C; c0 += 2) {
        const int c1 = min(c0 + 1, C - 1);
        const float4* row0 = reinterpret_cast<const float4*>(cb + c0 * pitch);
        const float4* row1 = reinterpret_cast<const float4*>(cb + c1 * pitch);
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int i = 0; i < GS / 4; ++i) {
          const float4 x = row0[i], y = row1[i];
          s0 = __fmaf_rn(k[4 * i], x.x, s0);
          s1 = __fmaf_rn(k[4 * i], y.x, s1);
          s0 = __fmaf_rn(k[4 * i + 1], x.y, s0);
          s1 = __fmaf_rn(k[4 * i + 1], y.y, s1);
          s0 = __fmaf_rn(k[4 * i + 2], x.z, s0);
          s1 = __fmaf_rn(k[4 * i + 2], y.z, s1);
          s0 = __fmaf_rn(k[4 * i + 3], x.w, s0);
          s1 = __fmaf_rn(k[4 * i + 3], y.w, s1);
        }
        const int v0 = ordered(s0), v1 = ordered(s1);
        if (v0 > best) { best = v0; code = c0; }
        if (v1 > best) { best = v1; code = c1; }
      }
    }
    return code;
  }
#pragma unroll 1
  for (int c0 = 0; c0 < C; c0 += 32 * kRows) {
    float x[kRows][GS];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {  // (past the end the last one again: the first lane of equal sums counts)
      const float4* row = reinterpret_cast<const float4*>(cb + min(c0 + 32 * r + lane, C - 1) * pitch);
#pragma unroll
      for (int i = 0; i < GS / 4; ++i) {
        const float4 v = row[i];
        x[r][4 * i] = v.x; x[r][4 * i + 1] = v.y; x[r][4 * i + 2] = v.z; x[r][4 * i + 3] = v.w;
      }
    }
#pragma unroll 1
    for (unsigned left = todo; left; left &= left - 1) {
      const int src = __ffs((int)left) - 1;
      float s[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) s[r] = 0.f;
#pragma unroll
      for (int d = 0; d < GS; ++d) {
        const float q = __shfl_sync(0xffffffffu, k[d], src);
#pragma unroll
        for (int r = 0; r < kRows; ++r) s[r] = __fmaf_rn(q, x[r][d], s[r]);
      }
      const int v0 = ordered(s[0]), v1 = kRows > 1 ? ordered(s[kRows - 1]) : v0;
      const int top = __reduce_max_sync(0xffffffffu, max(v0, v1));
      const unsigned in0 = __ballot_sync(0xffffffffu, v0 == top), in1 = __ballot_sync(0xffffffffu, v1 == top);
      const int at = c0 + (in0 ? __ffs((int)in0) - 1 : 31 + __ffs((int)in1));
      if (lane == src && top > best) { best = top; code = at; }
    }
  }
  return code;
}

// ---- operand of the centroids -----------------------------------------------------------------
// Tier slots searched together, at most kSumCols columns of sums at a time (a pass).  Columns of a pass:
// first half of the slice (the 16-dim slots' centroids side by side), second half, then the 32-dim slots.
// Shared memory: per pass, slice and part (hi, lo) 32-byte rows of 16 dims: first half, second half, and per 32-dim
// slot both halves; K-major without swizzle (8-row groups 256 bytes apart, 8-dim groups 128).
struct SearchPlan {
  int n_pass;
  int first[SPHKV_MAX_TIER_SLOTS + 1];  // pass p searches the slots list[first[p]] .. list[first[p + 1] - 1]
  int list[SPHKV_MAX_TIER_SLOTS];
  int n16[SPHKV_MAX_TIER_SLOTS];        // per pass: columns of a half, a multiple of 16
  int rows[SPHKV_MAX_TIER_SLOTS];       // per pass: operand rows of a slice and part
  int base[SPHKV_MAX_TIER_SLOTS];       // per pass: byte offset of its operand
  int col[SPHKV_MAX_TIER_SLOTS];        // per slot: first column, of a half (g 16) or of the pass (g 32)
  int row[SPHKV_MAX_TIER_SLOTS];        // per slot: first operand row (g 16: of the first half)
  int bytes;
};
__host__ __device__ inline int pad16(int n) { return (n + 15) & ~15; }

// slots whose bit is set in `wanted`
__host__ __device__ inline SearchPlan plan_search(const sphkv_tiers& t, int dh, unsigned wanted) {
  SearchPlan p = {};
  int n = 0;
  for (int s = 0; s < t.n_slots; ++s)
    if ((wanted >> s) & 1u) p.list[n++] = s;
  int i = 0;
  while (i < n) {
    const int ps = p.n_pass++;
    p.first[ps] = i;
    p.base[ps] = p.bytes;
    int c16 = 0, c32 = 0, last = i;
    for (; last < n; ++last) {  // as many slots as fit
      const int s = p.list[last], C = 1 << t.bits[s];
      const int a = c16 + (t.g[s] == 16 ? C : 0), b = c32 + (t.g[s] == 32 ? pad16(C) : 0);
      if (last > i && 2 * pad16(a) + b > kSumCols) break;
      c16 = a;
      c32 = b;
    }
    p.n16[ps] = pad16(c16);
    int at = 0, col32 = 2 * p.n16[ps], row32 = 2 * p.n16[ps];
    for (; i < last; ++i) {
      const int s = p.list[i], C = 1 << t.bits[s];
      if (t.g[s] == 16) {
        p.col[s] = p.row[s] = at;
        at += C;
      } else {
        p.col[s] = col32;
        p.row[s] = row32;
        col32 += pad16(C);
        row32 += 2 * pad16(C);
      }
    }
    p.rows[ps] = row32;
    p.bytes += row32 * 32 * 2 * (dh / 32);
  }
  p.first[p.n_pass] = n;
  return p;
}

// The operand and the largest norms of a KV head's centroids, by all threads of the CTA (between barriers of its own);
// most[slot * 8 + group] = max |c| of the group, NaN outside 2^-30 .. 2^30.  Four dims of a centroid at a time, so that
// loads are whole lines and many are in flight: a CTA does nothing else meanwhile.
__device__ __forceinline__ void stage_centroids(const SearchPlan& pl, const sphkv_tiers& t, const float* codebooks, int head, int dh,
                                                uint8_t* op, float* most) {
  if (threadIdx.x < SPHKV_MAX_TIER_SLOTS * 8) most[threadIdx.x] = 0.f;
  __syncthreads();
  for (int ps = 0; ps < pl.n_pass; ++ps) {
    for (int li = pl.first[ps]; li < pl.first[ps + 1]; ++li) {
      const int s = pl.list[li], bits = t.bits[s], qs = t.g[s] == 16 ? 2 : 3;  // log2 of a centroid's quads
      const int total = ((dh >> (qs + 2)) << bits) << qs, part = pl.rows[ps] * 32;
      const float* src = codebooks + ((int64_t)(head * t.n_slots + s) * t.G_max) * t.C_max * t.g_max;
#pragma unroll 4
      for (int i = threadIdx.x; i < total; i += kSearchThreads) {  // (a multiple of 32: whole warps)
        const int q = i & ((1 << qs) - 1), c = (i >> qs) & ((1 << bits) - 1), gam = i >> (qs + bits);
        const float4 x = __ldg(reinterpret_cast<const float4*>(src + ((int64_t)gam * t.C_max + c) * t.g_max) + q);
        // operand row of the centroid: slice, half / 16-dim part (a block of rows starts on a multiple of 16, so a row's place
        // follows from its number)
        const int slice = qs == 2 ? gam >> 1 : gam;
        const int r = qs == 2 ? (gam & 1) * pl.n16[ps] + pl.row[s] + c : pl.row[s] + (q >> 2) * pad16(1 << bits) + c;
        uint8_t* to = op + pl.base[ps] + slice * 2 * part + (r >> 3) * 256 + (r & 7) * 16 + ((q >> 1) & 1) * 128 + (q & 1) * 8;
        uint2 hi, lo;
        split_bf16x2(x.x, x.y, hi.x, lo.x);
        split_bf16x2(x.z, x.w, hi.y, lo.y);
        *reinterpret_cast<uint2*>(to) = hi;
        *reinterpret_cast<uint2*>(to + part) = lo;
        float nsq = (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w);
        for (int o = 1; o < 1 << qs; o <<= 1) nsq += __shfl_xor_sync(0xffffffffu, nsq, o);
        // norms are not negative: their bit patterns order as integers, a NaN above infinity.  Lanes of one group first
        int m = __float_as_int(nsq) & 0x7fffffff;
        const int lanes = min(32, 1 << (qs + bits));
        for (int o = 1 << qs; o < lanes; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((i & (lanes - 1)) == 0) atomicMax(reinterpret_cast<int*>(most + s * 8 + gam), m);
      }
    }
  }
  fence_async_smem();
  __syncthreads();
  if (threadIdx.x < SPHKV_MAX_TIER_SLOTS * 8) {
    const float nsq = most[threadIdx.x];
    most[threadIdx.x] = nsq >= 8.6736174e-19f && nsq <= 1.1529215e18f ? sqrtf(nsq) : __int_as_float(0x7fc00000);
  }
  __syncthreads();
}

// The products of one slice and pass, issued by one thread: sums at column `sums`, key pairs at column `keys` of the
// group's tensor memory, operand at shared address `op` (the slice's hi part).  `lows`: the keys have a lo part.
__device__ __forceinline__ void issue_products(const SearchPlan& pl, const sphkv_tiers& t, int ps, uint32_t sums, uint32_t keys,
                                               uint32_t op, bool lows) {
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);  // fp32 sums, bf16 x bf16, 128 rows
  const uint32_t lo_part = pl.rows[ps] * 2;  // 16-byte units
  auto product = [&](uint32_t d, int half, uint32_t b, int n, bool more) {
    const uint32_t idesc = kIdesc | ((uint32_t)(n >> 3) << 17);
    const uint64_t hi = smem_desc(0, 128, 256, 0) + b, lo = smem_desc(0, 128, 256, 0) + (b + lo_part);
    mma_ts(d, keys + 8 * half, hi, idesc, more);
    if (lows) mma_ts(d, keys + 16 + 8 * half, hi, idesc, true);
    mma_ts(d, keys + 8 * half, lo, idesc, true);
    if (lows) mma_ts(d, keys + 16 + 8 * half, lo, idesc, true);
  };
  const int n16 = pl.n16[ps];
  if (n16 > 0)
    for (int half = 0; half < 2; ++half) product(sums + half * n16, half, (op >> 4) + half * n16 * 2, n16, false);
  for (int li = pl.first[ps]; li < pl.first[ps + 1]; ++li) {
    const int s = pl.list[li], n = pad16(1 << t.bits[s]);
    if (t.g[s] != 32) continue;
    for (int half = 0; half < 2; ++half) product(sums + pl.col[s], half, (op >> 4) + (pl.row[s] + half * n) * 2, n, half > 0);
  }
}

// One or two rows of sums with 1 << bits columns (1 .. 6), first into registers, then searched: what lies between them runs
// while the tensor cores fill the columns again
struct RowSums {
  float a[64], b[64];
};
__device__ __forceinline__ void load_sums(RowSums& v, uint32_t addr_a, uint32_t addr_b, int bits, bool two) {
  auto run = [&](auto n) {
    constexpr int C = decltype(n)::value;
    float(&a)[C] = reinterpret_cast<float(&)[C]>(v.a);
    float(&b)[C] = reinterpret_cast<float(&)[C]>(v.b);
    tmem_ld_row<C>(addr_a, a);
    if (two) tmem_ld_row<C>(addr_b, b);
  };
  if (bits == 6)
    run(std::integral_constant<int, 64>());
  else if (bits == 5)
    run(std::integral_constant<int, 32>());
  else
    run(std::integral_constant<int, 16>());
  tmem_wait_ld();
}
template <int C>
__device__ __forceinline__ bool nearest_in(const float (&v)[64], float norm, float most, int& code) {
  return nearest_column<C>(reinterpret_cast<const float(&)[C < 16 ? 16 : C]>(v), norm, most, code);
}
__device__ __forceinline__ void search_sums(const RowSums& v, int bits, bool two, float norm_a, float norm_b, float most_a, float most_b,
                                            int& code_a, int& code_b, bool& sure_a, bool& sure_b) {
  auto run = [&](auto n) {
    constexpr int C = decltype(n)::value;
    sure_a = nearest_in<C>(v.a, norm_a, most_a, code_a);
    if (two) sure_b = nearest_in<C>(v.b, norm_b, most_b, code_b);
  };
  code_b = 0;
  sure_b = true;
  switch (bits) {
    case 6: run(std::integral_constant<int, 64>()); break;
    case 5: run(std::integral_constant<int, 32>()); break;
    case 4: run(std::integral_constant<int, 16>()); break;
    case 3: run(std::integral_constant<int, 8>()); break;
    case 2: run(std::integral_constant<int, 4>()); break;
    default: run(std::integral_constant<int, 2>()); break;
  }
}

}  // namespace sphkv
