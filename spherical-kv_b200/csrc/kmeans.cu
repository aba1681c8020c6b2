// Assignment + accumulation step of spherical k-means, the inner loop of codebook training
// (codebooks/generate.py:47-58): sims = U @ centers^T, assigns = argmax, per-cluster vector
// sums and counts.  The similarity search is the one of the page encoder: the dot product
// of a point with a centroid is an fp32 fma chain over d = 0..g-1 starting from 0, centroids
// are visited in ascending order and the first maximum wins (torch.argmax convention) -- found on the tensor cores
// and settled by the chains where that does not decide (search.cuh).
//
// The accumulation uses no float atomics and no barrier until the end: every warp keeps sums of its own in
// shared memory, 32 / D sets of [K][D] (`ways`; fewer when they would not fit), and walks its points D lanes to a row
// -- lane = dimension, one add per row and lane, the rows as they were staged -- so lanes never meet in an address.  At the
// end the warps' sets are added up and every CTA adds its sums to the output with float atomics, in no fixed order.
// Sums agree to rounding, as with index_add_ on a GPU; assignments and counts are exact.
#include <algorithm>

#include "search.cuh"

namespace sphkv {

// points per thread: 4 (2 for 32-dim points) keeps the kernel at two CTAs per SM
__host__ __device__ constexpr int pts_for(int d) { return d >= 32 ? 2 : 4; }

// Few centroids, and some numbers of points (see the rule at the launch): the chains on the fp32 pipe.  A CTA takes passes of 32 * pts_for(D) points per
// warp; its warps walk them without meeting; a warp's rows are turned through a 32-row tile for the adds.  Bound: fp32 FMA
// issue, then the shared-memory adds.
template <int D, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 2) kmeans_chains_kernel(
    const float* __restrict__ U, int64_t N, const float* __restrict__ centers, int K,
    int32_t* __restrict__ assigns, float* __restrict__ best_sim, float* __restrict__ sums,
    int32_t* __restrict__ counts, int ways) {
  constexpr int kPts = pts_for(D);
  constexpr int kWarpPts = 32 * kPts;           // points of a warp per pass
  extern __shared__ __align__(16) float sm[];
  constexpr int threads = 32 * WARPS;
  float* c_s = sm;                                            // [K][D] centres
  float* sum_s = sm + K * D;                                  // [warps][ways][K][D] sums
  int* cnt_s = reinterpret_cast<int*>(sum_s + WARPS * ways * K * D);     // [K] counts of this CTA
  uint8_t* code_s = reinterpret_cast<uint8_t*>(cnt_s + K);               // [warps][32]
  for (int i = threadIdx.x; i < K * D; i += threads) c_s[i] = centers[i];
  for (int i = threadIdx.x; i < WARPS * ways * K * D; i += threads) sum_s[i] = 0.f;
  for (int i = threadIdx.x; i < K; i += threads) cnt_s[i] = 0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* my_codes = code_s + warp * 32;
  // 32 rows of points, 16-byte chunk q of row p at chunk q ^ turn(p): neither the row-per-lane stores nor the
  // dimension-per-lane loads meet in a bank
  float* tile = reinterpret_cast<float*>(sm + K * D + WARPS * ways * K * D + ((K + 3) & ~3) + WARPS * 8) + warp * 32 * D;
  auto turn = [](int p) { return (p >> (D == 32 ? 0 : D == 16 ? 1 : 2)) & (D / 4 - 1); };
  // adding: lane = (way, dimension); with one way the first D lanes work
  const int dim = lane & (D - 1), way = lane / D;
  const bool adds = way < ways;
  float* my_sums = sum_s + ((int64_t)warp * ways + (adds ? way : 0)) * K * D + dim;

  const int64_t stride = (int64_t)gridDim.x * WARPS * kWarpPts;
  for (int64_t base = ((int64_t)blockIdx.x * WARPS + warp) * kWarpPts; base < N; base += stride) {
    float u[kPts][D];
    bool live[kPts];
#pragma unroll
    for (int h = 0; h < kPts; ++h) {
      const int64_t idx = base + lane + 32 * h;
      live[h] = idx < N;
      if (live[h]) {
        const float4* src = reinterpret_cast<const float4*>(U + idx * D);
#pragma unroll
        for (int q = 0; q < D / 4; ++q) {
          const float4 v = __ldg(src + q);
          u[h][4 * q] = v.x; u[h][4 * q + 1] = v.y; u[h][4 * q + 2] = v.z; u[h][4 * q + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < D; ++i) u[h][i] = 0.f;
      }
    }
    float best[kPts];
    int code[kPts];
#pragma unroll
    for (int h = 0; h < kPts; ++h) { best[h] = -INFINITY; code[h] = 0; }
    SPHKV_UNROLL_SEARCH
    for (int c = 0; c < K; ++c) {
      const float4* row = reinterpret_cast<const float4*>(c_s + c * D);
      float acc[kPts];
#pragma unroll
      for (int h = 0; h < kPts; ++h) acc[h] = 0.f;
#pragma unroll
      for (int q = 0; q < D / 4; ++q) {
        const float4 v = row[q];
#pragma unroll
        for (int h = 0; h < kPts; ++h) {
          acc[h] = __fmaf_rn(u[h][4 * q], v.x, acc[h]);
          acc[h] = __fmaf_rn(u[h][4 * q + 1], v.y, acc[h]);
          acc[h] = __fmaf_rn(u[h][4 * q + 2], v.z, acc[h]);
          acc[h] = __fmaf_rn(u[h][4 * q + 3], v.w, acc[h]);
        }
      }
#pragma unroll
      for (int h = 0; h < kPts; ++h)
        if (acc[h] > best[h]) { best[h] = acc[h]; code[h] = c; }
    }
#pragma unroll
    for (int h = 0; h < kPts; ++h) {
      const int64_t idx = base + lane + 32 * h;
      __syncwarp();  // the adds before have read the tile
      my_codes[lane] = (uint8_t)code[h];
#pragma unroll
      for (int q = 0; q < D / 4; ++q)
        *reinterpret_cast<float4*>(tile + lane * D + 4 * (q ^ turn(lane))) =
            make_float4(u[h][4 * q], u[h][4 * q + 1], u[h][4 * q + 2], u[h][4 * q + 3]);
      if (live[h]) {
        assigns[idx] = code[h];
        if (best_sim != nullptr) best_sim[idx] = best[h];
        atomicAdd(&cnt_s[code[h]], 1);
      }
      __syncwarp();
      if (adds) {  // rows past the end are zero and add nothing
        for (int p0 = 0; p0 < 32; p0 += 8 * ways) {
          float v[8];
          int c[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int p = p0 + e * ways + way;
            v[e] = tile[p * D + 4 * ((dim >> 2) ^ turn(p)) + (dim & 3)];
            c[e] = my_codes[p];
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) my_sums[c[e] * D] += v[e];
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < K * D; i += threads) {
    float t = 0.f;
    for (int w = 0; w < WARPS * ways; ++w) t += sum_s[(int64_t)w * K * D + i];
    if (t != 0.f) atomicAdd(sums + i, t);
  }
  for (int i = threadIdx.x; i < K; i += threads)
    if (cnt_s[i] != 0) atomicAdd(counts + i, cnt_s[i]);
}

template <int D, int WARPS = 8>
static int launch_chains(const float* U, int64_t N, const float* centers, int K, int32_t* assigns, float* best_sim, float* sums,
                         int32_t* counts, int sms, cudaStream_t st) {
  // a set of sums for every D lanes of a warp, or for fewer of them, while two CTAs fit an SM: with d 8 and K 128 two
  // sets fit where four do not (1M points: 86.4 us with one set, 80.4 with two)
  auto bytes = [&](int ways) {
    return ((size_t)K * D * (1 + WARPS * ways) + ((K + 3) & ~3) + WARPS * 8 + WARPS * 32 * D) * sizeof(float);
  };
  int ways = 32 / D;
  while (ways > 1 && bytes(ways) > 110 * 1024) ways >>= 1;
  const size_t smem = bytes(ways);
  // eight warps' sums are more than a CTA can have from K 173 on at d 32: seven (a runtime warp count cost every
  // size 1 to 4 %)
  if constexpr (WARPS == 8 && D == 32)
    if (smem > 227 * 1024) return launch_chains<D, 7>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st);
  static SmemOptIn opt_in;
  if (int rc = ensure_dynamic_smem(opt_in, (const void*)kmeans_chains_kernel<D, WARPS>, (int)smem, "kmeans_assign")) return rc;
  const int64_t pass = (int64_t)32 * WARPS * pts_for(D);
  const int64_t ctas = std::min<int64_t>((N + pass - 1) / pass, (int64_t)sms * (smem <= 110 * 1024 ? 2 : 1));
  kmeans_chains_kernel<D, WARPS><<<(unsigned)ctas, 32 * WARPS, smem, st>>>(U, N, centers, K, assigns, best_sim, sums, counts, ways);
  return check_launch("kmeans_chains_kernel");
}

// ---- search on the tensor cores ----
struct KmeansArgs {
  const float* U;
  int64_t N;
  const float* centers;
  int K;
  int32_t* assigns;
  float* best_sim;
  float* sums;
  int32_t* counts;
  int ways;        // sets of sums per warp
  int cols;        // tensor memory columns of a group
  int sum_cols;    // K rounded up to 16
  int off_centers, off_sums, off_points, off_small;  // byte offsets in shared memory (the centroids' operand at 0)
};

// batches of 128 points in flight per group, the one whose rows are being added included
__host__ __device__ constexpr int kmeans_stages(int d) { return d >= 32 ? 3 : 4; }
__host__ __device__ constexpr int kmeans_key_cols(int d) { return d >= 32 ? 32 : 16; }  // hi | lo of a point
constexpr int kKmeansGroups = 3;
// floats from one centroid to the next in shared memory: lanes that read rows of their own spread over all banks
__host__ __device__ constexpr int kmeans_pitch(int d) { return d + 4; }

__device__ __forceinline__ float lds_f1(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

// Three products, without lo * lo (2^-16 at most), and a lead that covers that too: a point's products are waited for, its chains are
// cheap.  4M points, K 64, with the fourth product and the smaller lead of search.cuh / so: 16 dims 149.9 / 149.1 us, 32 dims 263 / 258.
constexpr float kPointLead = 5.f / 65536.f;
static_assert(2 * (2 * kPairError + 1. / (1 << 16) + 6 * kSumError + kChainError + kRestError) < kPointLead, "the lead covers both sums' errors");

// The vote of search.cuh with the columns above t as bits, up to 24 to a float (exact sums): where there are more than one, it says
// which the chains have to decide between.  1M points of 16 dims, K 64, all centroids for an open point before / now / the chains'
// kernel: random 45 / 46 / 72 us, a tenth of the points' mean as spread 79 / 53 / 72, zeros 125 / 50 / 72, all centroids equal
// 123 / 123 / 72.  (The code cache's kernel has no registers for these.)
template <int C>
struct Leaders {
  static constexpr int kParts = (C + 23) / 24;
  float part[kParts];  // bit c - 24 i of part i: column c is above t, if t fits
};
template <int C>
__device__ __forceinline__ void find_leaders(const float (&v)[C < 16 ? 16 : C], const Lead& l, Leaders<C>& who) {
  constexpr int kSums = Leaders<C>::kParts > 1 ? 2 : 4;  // chains of a part
  float sum[Leaders<C>::kParts][kSums] = {};
#pragma unroll
  for (int c = 0; c < C; ++c) {
    float& to = sum[c / 24][c & (kSums - 1)];
    to = __fmaf_rn(__saturatef(__fmaf_rn(v[c], l.scale, l.shift)), (float)(1 << c % 24), to);
  }
#pragma unroll
  for (int i = 0; i < Leaders<C>::kParts; ++i) {
    if constexpr (kSums == 4)
      who.part[i] = (sum[i][0] + sum[i][1]) + (sum[i][2] + sum[i][3]);
    else
      who.part[i] = sum[i][0] + sum[i][1];
  }
}
// one leader: one part that is not 0 (their sum is the largest of them: parts are whole and below 2^24), and it a power of two,
// whose exponent is the leader's number
template <int C>
__device__ __forceinline__ bool one_leader(const Leaders<C>& who, int& code) {
  float one = who.part[0];
  bool single = true;
  if constexpr (Leaders<C>::kParts == 2) {
    single = who.part[0] + who.part[1] == fmaxf(who.part[0], who.part[1]);
    one = __fmaf_rn(who.part[1], 16777216.f, one);
  } else if constexpr (Leaders<C>::kParts == 3) {
    single = (who.part[0] + who.part[1]) + who.part[2] == max3(who.part[0], who.part[1], who.part[2]);
    one = __fmaf_rn(who.part[2], 281474976710656.f, __fmaf_rn(who.part[1], 16777216.f, one));
  }
  code = (__float_as_int(one) >> 23) - 127;
  return single && (__float_as_int(one) & 0x7fffff) == 0;
}
// those columns, or all where the sums do not say
template <int C>
__device__ __forceinline__ uint64_t open_columns(const Leaders<C>& who, bool all) {
  if (all) return ~0ull >> (64 - C);
  uint64_t open = 0;
#pragma unroll
  for (int i = 0; i < Leaders<C>::kParts; ++i) open |= (uint64_t)(uint32_t)who.part[i] << (24 * i);
  return open;
}

// The chains of N centroids side by side
template <int N, int GS>
__device__ __forceinline__ void chains(const float (&k)[GS], const float* __restrict__ cb, int pitch, const int (&c)[N], float (&sum)[N]) {
#pragma unroll
  for (int j = 0; j < N; ++j) sum[j] = 0.f;
#pragma unroll
  for (int i = 0; i < GS / 4; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float4 x = *reinterpret_cast<const float4*>(cb + c[j] * pitch + 4 * i);
      sum[j] = __fmaf_rn(k[4 * i], x.x, sum[j]);
      sum[j] = __fmaf_rn(k[4 * i + 1], x.y, sum[j]);
      sum[j] = __fmaf_rn(k[4 * i + 2], x.z, sum[j]);
      sum[j] = __fmaf_rn(k[4 * i + 3], x.w, sum[j]);
    }
}
// the first maximum of all C (past the end the last one again, which is not larger than itself)
template <int GS>
__device__ __forceinline__ int walk_all(const float (&k)[GS], const float* __restrict__ cb, int pitch, int C) {
  constexpr int N = GS < 32 ? 4 : 2;
  float best = -INFINITY;
  int code = 0;
#pragma unroll 1
  for (int c0 = 0; c0 < C; c0 += N) {
    int c[N];
    float sum[N];
#pragma unroll
    for (int j = 0; j < N; ++j) c[j] = min(c0 + j, C - 1);
    chains(k, cb, pitch, c, sum);
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (sum[j] > best) { best = sum[j]; code = c[j]; }
  }
  return code;
}
// the same among the columns c0 + (bits of `open`), two at a time (bits ascend: the first maximum stays the first)
template <int GS, typename Bits>
__device__ __forceinline__ void walk_open(const float (&k)[GS], const float* __restrict__ cb, int pitch, int c0, Bits open, float& best, int& code) {
#pragma unroll 1
  while (open) {
    int c[2];
    float sum[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int at = sizeof(Bits) == 8 ? __ffsll((long long)open) : __ffs((int)open);
      c[j] = at > 0 ? c0 + at - 1 : c[0];
      open &= open - 1;
    }
    chains(k, cb, pitch, c, sum);
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (sum[j] > best) { best = sum[j]; code = c[j]; }
  }
}
// a lane's point k, with the columns `open`
template <int GS>
__device__ __forceinline__ int settle_point(const float (&k)[GS], const float* __restrict__ cb, int pitch, int C, uint64_t open, int code) {
  if (open && first_wins(k, cb)) {
    code = 0;
    open = 0;
  }
  if (__any_sync(0xffffffffu, __popcll(open) > 8)) {
    if (open) code = walk_all(k, cb, pitch, C);
  } else if (open) {
    float best = -INFINITY;
    code = 0;
    walk_open(k, cb, pitch, 0, open, best, code);
  }
  return code;
}

// Bound: latency -- twelve warps an SM, each with a chain of tensor memory, shared-memory adds and a barrier per batch (58 % of
// issue slots, L1 and shared memory 56 %, DRAM 22 %).  4M points, d 16, K 64: 254 us with the chains, 170 here, 148 without bank
// conflicts on the winners.
// A CTA has up to three search groups (four warps, thread = point = lane of tensor memory), each striding over batches
// of 128 points; a warp stages, splits, searches and adds its 32 points by itself and meets the group's other warps
// once per batch, before the products.
template <int D>
__global__ void __launch_bounds__(kKmeansGroups * 128, 1) kmeans_search_kernel(const __grid_constant__ KmeansArgs a) {
  constexpr int kStages = kmeans_stages(D), kKeys = kmeans_key_cols(D), kParts = D >= 32 ? 2 : 1;
  constexpr int kRowChunks = D / 4;  // 16-byte chunks of a point
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int group = warp >> 2, w = warp & 3, groups = blockDim.x >> 7, K = a.K;
  constexpr int kPitch = kmeans_pitch(D);
  float* c_s = reinterpret_cast<float*>(smem + a.off_centers);           // [K][kPitch]
  float* sum_s = reinterpret_cast<float*>(smem + a.off_sums);            // [warps][ways][K][D]
  int* cnt_s = reinterpret_cast<int*>(smem + a.off_small);               // [K]
  int* most_s = cnt_s + ((K + 3) & ~3);                                  // largest |c|^2
  const uint32_t bars = smem_u32(most_s + 2), bar = bars + 8 * group;
  volatile uint32_t* tmem_word = reinterpret_cast<volatile uint32_t*>(most_s + 2 + 2 * kKmeansGroups);
  const uint32_t points = smem_u32(smem + a.off_points) + warp * (kStages * 32 * D * 4);
  // chunk q of row p is stored at chunk q ^ turn(p): neither row-per-lane nor dimension-per-lane accesses meet in a bank
  auto turn = [](int p) { return (p >> (D == 32 ? 0 : D == 16 ? 1 : 2)) & (kRowChunks - 1); };

  const int64_t stride = (int64_t)gridDim.x * groups * 128;
  const int64_t first = ((int64_t)blockIdx.x * groups + group) * 128;
  int64_t fetch_at = first + 32 * w;
  int fetch_stage = 0;
  auto fetch = [&]() {  // the warp's 32 rows of the next batch
    if (fetch_at - 32 * w < a.N) {  // the group's batch; rows past the end are zero
      const float* src = a.U + fetch_at * D;
      const int chunks = (int)max((int64_t)0, min((int64_t)32, a.N - fetch_at)) * kRowChunks;
      const uint32_t dst = points + fetch_stage * (32 * D * 4);
#pragma unroll
      for (int i = 0; i < kRowChunks; ++i) {
        const int c = lane + 32 * i, p = c / kRowChunks, q = c % kRowChunks;
        const bool in = c < chunks;
        cp_async_16_zfill(dst + p * (D * 4) + (q ^ turn(p)) * 16, in ? src + 4 * c : a.U, in ? 16 : 0);
      }
    }
    cp_async_commit();
    fetch_at += stride;
    fetch_stage = fetch_stage + 1 == kStages ? 0 : fetch_stage + 1;
  };
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) fetch();

  if (warp == 0) tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_word)), 512);
  if ((int)threadIdx.x < groups) mbar_init(bars + 8 * threadIdx.x, 1);
  if (threadIdx.x == 0) *most_s = 0;
  for (int i = threadIdx.x; i < K * D; i += blockDim.x) c_s[i / D * kPitch + i % D] = a.centers[i];
  for (int i = threadIdx.x; i < (int)(blockDim.x >> 5) * a.ways * K * D; i += blockDim.x) sum_s[i] = 0.f;
  for (int i = threadIdx.x; i < K; i += blockDim.x) cnt_s[i] = 0;
  __syncthreads();
  // operand of the centroids: per part (hi, lo) and 16 dims, rows of 32 bytes, 8-row groups 256 bytes apart, 8-dim
  // groups 128; points of 8 dims are padded with zeros
  const int part_bytes = a.sum_cols * 32 * kParts;
  for (int i = threadIdx.x; i < K * kParts; i += blockDim.x) {
    const int c = i / kParts, kc = i % kParts;
    uint8_t* hi_at = smem + kc * a.sum_cols * 32 + (c >> 3) * 256 + (c & 7) * 16;
    uint32_t hi[8], lo[8];
    float nsq = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float x = 2 * e < D ? c_s[c * kPitch + 16 * kc + 2 * e] : 0.f, y = 2 * e < D ? c_s[c * kPitch + 16 * kc + 2 * e + 1] : 0.f;
      split_bf16x2(x, y, hi[e], lo[e]);
    }
    *reinterpret_cast<uint4*>(hi_at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(hi_at + 128) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
    *reinterpret_cast<uint4*>(hi_at + part_bytes) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    *reinterpret_cast<uint4*>(hi_at + part_bytes + 128) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
    if (kc == 0) {
      for (int e = 0; e < D; ++e) nsq += c_s[c * kPitch + e] * c_s[c * kPitch + e];
      atomicMax(most_s, __float_as_int(nsq) & 0x7fffffff);  // bit patterns order as integers, a NaN above infinity
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const float most_sq = __int_as_float(*most_s);
  const float most = most_sq >= 8.6736174e-19f && most_sq <= 1.1529215e18f ? sqrtf(most_sq) : __int_as_float(0x7fc00000);
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_word[0], 0);
  const uint32_t tmem = tmem_base + group * a.cols, my_rows = tmem + ((uint32_t)(32 * w) << 16);
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);  // fp32 sums, bf16 x bf16, 128 rows
  const uint32_t idesc = kIdesc | ((uint32_t)(a.sum_cols >> 3) << 17);
  const uint64_t op = smem_desc(smem_u32(smem), 128, 256, 0);

  float norm_n = 0.f;
  int conv_stage = 0, keys = 0;
  auto convert = [&]() {  // the next staged batch's rows as bf16 pairs in tensor memory
    cp_async_wait<kStages - 2>();
    __syncwarp();
    const uint32_t src = points + conv_stage * (32 * D * 4) + lane * (D * 4);
    float k[D < 16 ? 16 : D];
#pragma unroll
    for (int q = 0; q < kRowChunks; ++q) {
      const float4 v = lds_f4(src + ((q ^ turn(lane)) << 4));
      k[4 * q] = v.x; k[4 * q + 1] = v.y; k[4 * q + 2] = v.z; k[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int i = D; i < 16; ++i) k[i] = 0.f;
    float n0 = 0.f, n1 = 0.f;
#pragma unroll
    for (int i = 0; i < D; i += 2) { n0 = __fmaf_rn(k[i], k[i], n0); n1 = __fmaf_rn(k[i + 1], k[i + 1], n1); }
    norm_n = sqrtf(n0 + n1);
    constexpr int kWords = (D < 16 ? 16 : D) / 2;
    uint32_t hi[kWords], lo[kWords];
    split_pairs(k, hi, lo);
    const uint32_t dst = my_rows + a.sum_cols + keys * kKeys;
    if constexpr (kWords == 16) {
      tmem_st_x16(dst, hi);
      tmem_st_x16(dst + 16, lo);
    } else {
      tmem_st_x8(dst, hi);
      tmem_st_x8(dst + 8, lo);
    }
    tmem_wait_st();
    conv_stage = conv_stage + 1 == kStages ? 0 : conv_stage + 1;
  };
  ProductWaits waits;  // once one ran out the chains decide everything
  auto wait = [&](uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0; };
  auto products = [&]() {
    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
    if (w == 0 && !waits.lost) {
      tc_fence_after();
      if (elect_one()) {
        const uint32_t k0 = tmem + a.sum_cols + keys * kKeys;
#pragma unroll
        for (int kc = 0; kc < kParts; ++kc) {
          const uint64_t hi = op + (uint32_t)(kc * a.sum_cols * 2), lo = hi + (uint32_t)(part_bytes >> 4);
          mma_ts(tmem, k0 + 8 * kc, hi, idesc, kc > 0);
          mma_ts(tmem, k0 + kKeys / 2 + 8 * kc, hi, idesc, true);
          mma_ts(tmem, k0 + 8 * kc, lo, idesc, true);
        }
        mma_commit(bar);
      }
      __syncwarp();
    }
    keys ^= 1;
  };
  // adding: lane = (way, dimension); with one way the first D lanes work
  const int dim = lane & (D - 1), way = lane / D;
  const bool adds = way < a.ways;
  float* my_sums = sum_s + ((int64_t)warp * a.ways + (adds ? way : 0)) * K * D + dim;

  if (first < a.N) {
    convert();
    tc_fence_before();
    products();
  }
  int stage = 0;
  for (int64_t base = first; base < a.N; base += stride) {
    const float norm = norm_n;
    const bool more = base + stride < a.N;
    fetch();
    if (more) convert();
    waits.next(wait);
    tc_fence_after();
    const int64_t idx = base + 32 * w + lane;
    const bool live = idx < a.N;
    const uint32_t rows = points + stage * (32 * D * 4);
    auto load = [&](float (&k)[D]) {
#pragma unroll
      for (int q = 0; q < kRowChunks; ++q) {
        const float4 v = lds_f4(rows + lane * (D * 4) + ((q ^ turn(lane)) << 4));
        k[4 * q] = v.x; k[4 * q + 1] = v.y; k[4 * q + 2] = v.z; k[4 * q + 3] = v.w;
      }
    };
    int code;
    auto whole = [&](auto n) {  // all sums of a point at once
      constexpr int C = decltype(n)::value;
      float v[C < 16 ? 16 : C];
      Leaders<C> who;
      tmem_ld_row<C>(my_rows, v);
      tmem_wait_ld();
      const Lead l = lead_of(largest_of<C>(v), norm, most, kPointLead);
      find_leaders<C>(v, l, who);
      const bool unsure = live && !(one_leader<C>(who, code) && l.fit && !waits.lost);
      tc_fence_before();
      if (more) products();  // runs while this batch is added up
      if (__any_sync(0xffffffffu, unsure)) {
        float k[D];
        load(k);
        code = settle_point(k, c_s, kPitch, K, unsure ? open_columns<C>(who, waits.lost || !l.fit) : 0, code);
      }
    };
    if (K == 64) {
      whole(std::integral_constant<int, 64>());
    } else if (D == 32 && K == 16) {  // (points of fewer dims come with more centroids)
      whole(std::integral_constant<int, 16>());
    } else if (D == 32 && K == 8) {
      whole(std::integral_constant<int, 8>());
    } else {  // sixteen columns at a time, twice: the largest, then what comes near it
      float top = -INFINITY;
      auto columns = [&](int c0, float (&v)[16]) {
        tmem_ld_x16(my_rows + c0, v);
        tmem_wait_ld();
        if (c0 + 16 > K) {
#pragma unroll
          for (int c = 0; c < 16; ++c)
            if (c0 + c >= K) v[c] = -INFINITY;
        }
      };
      for (int c0 = 0; c0 < K; c0 += 16) {
        float v[16];
        columns(c0, v);
        top = fmaxf(top, largest_of<16>(v));
      }
      const Lead l = lead_of(top, norm, most, kPointLead);
      Leaders<16> who = {{0.f}};
      int base_of = 0;
      uint32_t blocks = 0;  // of sixteen columns, with some above t
      for (int c0 = 0, bit = 1; c0 < K; c0 += 16, bit <<= 1) {
        float v[16];
        columns(c0, v);
        Leaders<16> some;
        find_leaders<16>(v, l, some);
        if (some.part[0] != 0.f) { who = some; base_of = c0; blocks |= bit; }
      }
      const bool one = one_leader<16>(who, code) && l.fit && (blocks & (blocks - 1)) == 0;
      code += base_of;
      bool unsure = live && !(one && !waits.lost);
      if (__any_sync(0xffffffffu, unsure)) {
        float k[D];
        load(k);
        if (unsure && first_wins(k, c_s)) {
          code = 0;
          unsure = false;
        }
        bool walk = unsure && (waits.lost || !l.fit);
        int n_open = 0;
        float best = -INFINITY;
        for (uint32_t todo = __reduce_or_sync(0xffffffffu, unsure ? blocks : 0u); todo && !__any_sync(0xffffffffu, walk); todo &= todo - 1) {
          const int c0 = 16 * (__ffs((int)todo) - 1);
          float v[16];
          columns(c0, v);
          Leaders<16> some;
          find_leaders<16>(v, l, some);
          const uint32_t above = unsure ? (uint32_t)some.part[0] : 0u;
          n_open += __popc(above);
          walk = n_open > 32;  // all are as fast one after the other
          if (!__any_sync(0xffffffffu, walk)) walk_open(k, c_s, kPitch, c0, above, best, code);
        }
        if (__any_sync(0xffffffffu, walk) && unsure) code = walk_all(k, c_s, kPitch, K);
      }
      tc_fence_before();
      if (more) products();
    }
    if (!live) code = 0;
    if (live) {
      a.assigns[idx] = code;
      if (a.best_sim != nullptr) {  // the chain of the winner
        float s = 0.f;
        const float4* c = reinterpret_cast<const float4*>(c_s + code * kPitch);
#pragma unroll
        for (int q = 0; q < kRowChunks; ++q) {
          const float4 v = lds_f4(rows + lane * (D * 4) + ((q ^ turn(lane)) << 4)), x = c[q];
          s = __fmaf_rn(v.x, x.x, s);
          s = __fmaf_rn(v.y, x.y, s);
          s = __fmaf_rn(v.z, x.z, s);
          s = __fmaf_rn(v.w, x.w, s);
        }
        a.best_sim[idx] = s > -INFINITY ? s : -INFINITY;  // a point whose sums are all NaN has none: -inf, as in the chains' kernel
      }
      atomicAdd(&cnt_s[code], 1);
    }
    // rows past the end are zero and add nothing.  Two rows at a time: if they are of one cluster, the second sum
    // follows from the first
    const int at = code * D;
    for (int p0 = 0; p0 < 32; p0 += 8 * a.ways) {
      float v[8];
      int c[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int p = p0 + e * a.ways + (adds ? way : 0);
        c[e] = __shfl_sync(0xffffffffu, at, p & 31);
        v[e] = lds_f1(rows + p * (D * 4) + (((dim >> 2) ^ turn(p)) << 4) + (dim & 3) * 4);
      }
      if (adds) {
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const float s0 = my_sums[c[e]], s1 = my_sums[c[e + 1]];
          const float t0 = s0 + v[e], t1 = (c[e] == c[e + 1] ? t0 : s1) + v[e + 1];
          my_sums[c[e]] = t0;
          my_sums[c[e + 1]] = t1;
        }
      }
    }
    __syncwarp();
    stage = stage + 1 == kStages ? 0 : stage + 1;
  }
  if (w == 0) waits.leave(wait);
  cp_async_wait<0>();
  tc_fence_before();
  __syncthreads();
  for (int i = threadIdx.x; i < K * D; i += blockDim.x) {
    float t = 0.f;
    for (int s = 0; s < (int)(blockDim.x >> 5) * a.ways; ++s) t += sum_s[(int64_t)s * K * D + i];
    if (t != 0.f) atomicAdd(a.sums + i, t);
  }
  for (int i = threadIdx.x; i < K; i += blockDim.x)
    if (cnt_s[i] != 0) atomicAdd(a.counts + i, cnt_s[i]);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D>
static int launch_search(KmeansArgs a, int sms, cudaStream_t st) {
  a.sum_cols = (a.K + 15) & ~15;
  a.cols = a.sum_cols + 2 * kmeans_key_cols(D);
  const int set = a.K * D * 4, parts = D >= 32 ? 2 : 1;
  const int small = ((a.K + 3) & ~3) * 4 + 8 + 8 * kKmeansGroups + 16;
  auto bytes = [&](int groups, int ways) {
    a.off_centers = a.sum_cols * 32 * parts * 2;
    a.off_sums = a.off_centers + a.K * kmeans_pitch(D) * 4;
    a.off_points = a.off_sums + (4 * groups * ways * set + 15) / 16 * 16;
    a.off_small = a.off_points + 4 * groups * kmeans_stages(D) * 32 * D * 4;
    return a.off_small + small;
  };
  // as many groups as tensor memory and shared memory have room for, then as many sets of sums
  int groups = kKmeansGroups, ways = 1;
  while (groups > 1 && (groups * a.cols > 512 || bytes(groups, 1) > 227 * 1024)) --groups;
  for (int more = 32 / D; more > ways; more >>= 1)
    if (bytes(groups, more) <= 227 * 1024) ways = more;
  const int smem = bytes(groups, ways);
  a.ways = ways;
  static SmemOptIn opt_in;
  if (int rc = ensure_dynamic_smem(opt_in, (const void*)kmeans_search_kernel<D>, smem, "kmeans_assign")) return rc;
  const int64_t ctas = std::min<int64_t>((a.N + 128 * groups - 1) / (128 * groups), sms);
  kmeans_search_kernel<D><<<(unsigned)ctas, 128 * groups, smem, st>>>(a);
  return check_launch("kmeans_search_kernel");
}

}  // namespace sphkv

using namespace sphkv;

extern "C" int sphkv_kmeans_assign(const float* U, int64_t N, int32_t d, const float* centers, int32_t K,
                                   int32_t* assigns, float* best_sim, float* sums, int32_t* counts,
                                   void* stream) {
  SPHKV_REQUIRE(U && centers && assigns && sums && counts, SPHKV_E_ARG, "kmeans_assign: NULL pointer");
  SPHKV_REQUIRE(N >= 0 && (d == 8 || d == 16 || d == 32) && K >= 1 && K <= 256, SPHKV_E_ARG,
                "kmeans_assign: N=%lld d=%d (8, 16 or 32) K=%d (1..256)", (long long)N, d, K);
  SPHKV_REQUIRE((reinterpret_cast<uintptr_t>(U) & 15) == 0, SPHKV_E_ARG, "kmeans_assign: U must be 16-byte aligned");
  const int sms = sphkv_sm_count();
  SPHKV_REQUIRE(sms > 0, SPHKV_E_ARG, "kmeans_assign: cannot resolve the SM count");
  // the sizes the call takes (8 and 16: every K; 32: K up to 179); all of them fit with one group and one set of sums per warp
  const int per_pass = 256 * (d >= 32 ? 2 : 4) * 2;
  SPHKV_REQUIRE(K * d * 8 + (3 * K + 1) * 4 + per_pass <= 48 * 1024, SPHKV_E_LIMIT,
                "kmeans_assign: K=%d x d=%d is beyond the sizes it takes (K * d * 8 + 12 * K + %d <= 49152)", K, d, 4 + per_pass);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(float) * K * d, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(counts, 0, sizeof(int32_t) * K, st);
  if (e != cudaSuccess) {
    set_error("kmeans_assign: cudaMemsetAsync: %s", cudaGetErrorString(e));
    return (int)e;
  }
  if (N == 0) return SPHKV_OK;
  // The chains cost K fmas per value, the tensor cores hardly anything, but that kernel has fewer warps to hide the sums behind.
  // Chains / tensor cores in us, without similarities:
  //   d 8   4M points K 32 96 / 103, 48 125 / 115, 64 156 / 101, 256 540 / 512; 30000 points K 32 11.1 / 10.3, 48 12.4 / 10.8
  //   d 16  4M K 16 121 / 114 (36.9 / 36.2 of 1M; with similarities slower), 24 142 / 139, 32 162 / 128, 64 254 / 125;
  //         30000 K 32 14.4 / 11.8
  //   d 32  4M K 2 219 / 173, 8 249 / 146, 64 557 / 211, 179 1519 / 628; 4096 points K 2 12.1 / 10.4, 128 29.1 / 22.7
  // In between, where the chains are done in one round of blocks and this kernel begins its second or third, or has only one
  // search group (more than 224 centroids of 8 dims): d 8 150000 points K 48 13.1 / 14.4, 256 30.9 / 37.3 (500000: 89.6 / 82.1);
  // d 16 150000 K 32 14.6 / 16.2 (100000: 14.4 / 12.4); d 32 65536 K 4 12.3 / 14.4.
  const auto between = [&](int lo, int hi) { return N > (int64_t)sms * lo && N <= (int64_t)sms * hi; };
  const bool chains = d == 8    ? K < 48 || (K < 64 && between(768, 2048)) || (K > 224 && between(512, 2048))
                      : d == 16 ? K < 32 || (K < 48 && between(768, 1024))
                                : K <= 8 && between(384, 512);
  if (chains) {
    return d == 8    ? launch_chains<8>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st)
           : d == 16 ? launch_chains<16>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st)
                     : launch_chains<32>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st);
  }
  KmeansArgs a = {};
  a.U = U; a.N = N; a.centers = centers; a.K = K;
  a.assigns = assigns; a.best_sim = best_sim; a.sums = sums; a.counts = counts;
  return d == 8 ? launch_search<8>(a, sms, st) : d == 16 ? launch_search<16>(a, sms, st) : launch_search<32>(a, sms, st);
}
