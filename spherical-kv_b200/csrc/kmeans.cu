// Assignment + accumulation step of spherical k-means, the inner loop of codebook training
// (codebooks/generate.py:47-58): sims = U @ centers^T, assigns = argmax, per-cluster vector
// sums and counts.  The similarity search is the one of the page encoder: the dot product
// of a point with a centroid is an fp32 fma chain over d = 0..g-1 starting from 0, centroids
// are visited in ascending order and the first maximum wins (torch.argmax convention).
//
// One thread holds kPts points in registers and walks the centroids out of shared memory
// (one broadcast 16-byte load feeds 16 or 8 FMAs).  The accumulation uses no float atomics and no
// barrier until the end: every warp keeps sums of its own in shared memory, 32 / D sets of [K][D] (`ways`; fewer
// when they would not fit), and walks its points D lanes to a row -- lane = dimension, one add per row and lane, the rows
// turned through a 32-row tile of shared memory -- so lanes never meet in an address.  At the end the
// warps' sets are added up and every CTA adds its sums to the output with float atomics, in no fixed order.  Sums agree to rounding, as with index_add_ on a GPU; assignments and counts are
// exact.  Bound: fp32 FMA issue for K = 64, then the shared-memory adds.  4M points, d 16, K 64: 324 -> 254 us;
// K 16, 2.3M points: 95 -> 76 us (a counting sort per 1024 points with six barriers before).
#include <algorithm>

#include "common.cuh"

namespace sphkv {

// points per thread: 4 (2 for 32-dim points) keeps the kernel at two CTAs per SM
__host__ __device__ constexpr int pts_for(int d) { return d >= 32 ? 2 : 4; }

// a CTA takes passes of 32 * pts_for(D) points per warp; its warps walk them without meeting
template <int D, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 2) kmeans_assign_kernel(
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
static int launch_kmeans(const float* U, int64_t N, const float* centers, int K, int32_t* assigns, float* best_sim, float* sums,
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
    if (smem > 227 * 1024) return launch_kmeans<D, 7>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st);
  static SmemOptIn opt_in;
  if (int rc = ensure_dynamic_smem(opt_in, (const void*)kmeans_assign_kernel<D, WARPS>, (int)smem, "kmeans_assign")) return rc;
  const int64_t pass = (int64_t)32 * WARPS * pts_for(D);
  const int64_t ctas = std::min<int64_t>((N + pass - 1) / pass, (int64_t)sms * (smem <= 110 * 1024 ? 2 : 1));
  kmeans_assign_kernel<D, WARPS><<<(unsigned)ctas, 32 * WARPS, smem, st>>>(U, N, centers, K, assigns, best_sim, sums, counts, ways);
  return check_launch("kmeans_assign_kernel");
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
  // the sizes the call takes (8 and 16: every K; 32: K up to 179); all of them fit with one set of sums per warp
  const int per_pass = 256 * pts_for(d) * 2;
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
  return d == 8    ? launch_kmeans<8>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st)
         : d == 16 ? launch_kmeans<16>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st)
                   : launch_kmeans<32>(U, N, centers, K, assigns, best_sim, sums, counts, sms, st);
}
