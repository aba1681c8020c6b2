// Split-K angle-domain decode attention: work split, tile metadata and the kernel itself.
#pragma once
#include <type_traits>

#include "tcgen05.cuh"

namespace sphkv {

// Roles of the 16 warps: three teams of four (a team = the 128 TMEM lanes = 128 token rows), and a
// driver warp per team; the last warp allocates tensor memory.
constexpr int kTeams = 3;
constexpr int kTeamThreads = 4 * kTeams * 32, kDecodeThreads = kTeamThreads + 4 * 32;
constexpr int kMacroTiles = 8;   // 16-token tiles per macro tile (128 rows)
constexpr int kMetaRing = 64;    // tiles of metadata per team, refilled 32 at a time
// Macro tiles of page bytes per team.  Three when a tile's stage is small enough (int8 radii): a copy issued
// while the teams weigh macro tile k has to land before they finish rebuilding the first half of k + 1,
// which two stages leave no room for under load.
constexpr int kKStages = 3;
// Registers: the launch gives every thread 128; the drivers return theirs to the teams
// (3 * 152 + 56 = 4 * 128 per four warps).
constexpr int kTeamRegs = 152, kDriverRegs = 56;
static_assert(kTeams * kTeamRegs + kDriverRegs <= 4 * 128 && kTeams == 3, "register split exceeds the launch");
// tensor memory columns of a team: rebuilt keys (hi | lo), logits, output accumulator
constexpr int kColKeys = 0, kColLogits = 128, kColOut = 144, kTeamCols = 160, kTmemCols = 512;
static_assert(kKStages <= 3 && kMetaRing == 8 * kMacroTiles, "metadata is ready three macro tiles ahead");
static_assert(kTeams * kTeamCols <= kTmemCols, "tensor memory");

// One 16-token tile, computed by the driver for 32 tiles at a time (16 bytes in the metadata ring)
struct TileMeta {
  int phys;        // physical page id; -1 hole / invalid page, -2 no such tile
  uint32_t where;  // tokens of the tile, at most | tier slot << 8 | stage byte offsets: header << 12, theta << 16
                   // (bytes; 9 bits); (theta - page) >> 7 << 25; sub tile of the page << 28
  uint32_t rad;    // stage byte offset of the tile's first radius byte | (theta - page) & 127 << 9 |
                   // (radii - theta) << 16
  int poff;        // page offset in the byte pool
};
__device__ __forceinline__ int meta_tokens(const TileMeta& m) { return m.where & 0xFF; }
__device__ __forceinline__ int meta_slot(const TileMeta& m) { return (m.where >> 8) & 0x3; }
__device__ __forceinline__ uint32_t meta_hdr(const TileMeta& m) { return (m.where >> 12) & 0xF; }
__device__ __forceinline__ uint32_t meta_theta(const TileMeta& m) { return (m.where >> 16) & 0x1FF; }
__device__ __forceinline__ uint32_t meta_radius(const TileMeta& m) { return m.rad & 0x1FF; }
__device__ __forceinline__ int meta_sub(const TileMeta& m) { return m.where >> 28; }

struct DecodeArgs {
  alignas(64) CUtensorMap v_map;  // V pool as [dh / 64][pages * page_size rows][64], boxes of 16 rows, 128-byte swizzle
  sphkv_decode_params p;
  int cb_smem_off[SPHKV_MAX_TIER_SLOTS];  // byte offset of each slot's codebook in smem
  int cb_dup[SPHKV_MAX_TIER_SLOTS];       // 1: two copies at a 128-byte row pitch
  int cb_smem_bytes;
  int n_units;
  int n_ctas;
  int grp;
  int teams;             // teams in use: 3, fewer when large codebooks leave less shared memory
  int wide;              // byte pool and positions start on 16-byte boundaries
  int plan_in_kernel;    // every CTA derives the block prefix itself (n_units small enough)
  int32_t* pfx;
  uint32_t* spans;  // per unit, for the merge: first CTA with a partial row | number of them << 16
  float* rows;  // [(n_ctas + n_units)][8][dh + 2]
};

// shared-memory carve-up, shared by host and device: query operand; per team barriers, votes and reference maxima, two words of
// the CTA; per team in use V tiles, weights, K stages, metadata; per team in use statistics; then codebooks and the block
// prefix.  Everything a team touches per tile lies at a constant offset from two bases: addresses that depended on the number
// of teams were made again at every use, 110 of 755 instructions a tile.  The statistics are read at a merge only, and
// behind the teams they leave the rest of the head 1024 bytes: a byte more here is a byte less for teams and codebook copies.
constexpr int kBarStride = 96, kSmemTeamBars = kBarStride + 32 + 128 + 32;
constexpr int kSmemStats = 256;  // per team
__host__ __device__ constexpr int smem_q_bytes(int dh) { return dh / 16 * 512; }
__host__ __device__ constexpr int smem_head_bytes(int dh) { return smem_q_bytes(dh) + 1024; }
static_assert(kTeams * kSmemTeamBars + 16 <= 1024, "barrier block");
__host__ __device__ constexpr int smem_v_bytes(int dh) { return kMacroTiles * 16 * dh * 2; }
constexpr int kSmemP = kMacroTiles * 512;
constexpr int kSmemK = 3 * kMacroTiles * 384;  // (f16 radii: 2 x 512)
constexpr int kSmemMeta = kMetaRing * 16;
__host__ __device__ constexpr int smem_team_bytes(int dh) { return smem_v_bytes(dh) + kSmemP + kSmemK + kSmemMeta; }
static_assert(smem_team_bytes(64) % 1024 == 0 && smem_team_bytes(128) % 1024 == 0 && smem_head_bytes(64) % 1024 == 0 &&
                  smem_head_bytes(128) % 1024 == 0, "V tiles start on 1024 bytes");
__host__ __device__ constexpr int smem_fixed_bytes(int dh, int teams) { return smem_head_bytes(dh) + teams * (smem_team_bytes(dh) + kSmemStats); }
// room for the group shifts of a slot's codebook (see stage_codebooks)
constexpr int kCbShift = 128;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
// codebook rows only: they do not change while a segment is processed, so the load may be
// scheduled freely
__device__ __forceinline__ float4 lds128(uint32_t addr) {
  float4 v;
  asm("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ int lds_s8(uint32_t addr) {
  int v;
  asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ TileMeta lds_meta(uint32_t addr) {
  TileMeta m;
  uint32_t x, y;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(x), "=r"(m.where), "=r"(m.rad), "=r"(y) : "r"(addr));
  m.phys = (int)x; m.poff = (int)y;
  return m;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void sts_meta(uint32_t addr, const TileMeta& m) {
  sts128(addr, (uint32_t)m.phys, m.where, m.rad, (uint32_t)m.poff);
}
__device__ __forceinline__ void cta_barrier() { asm volatile("bar.sync 0;" ::: "memory"); }
__device__ __forceinline__ void teams_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kTeamThreads) : "memory"); }

// Frequencies of a lane (also the layout of the RoPE table): for loop index i (0 .. W/4 - 1) and lane quad
// member j (0 .. 3) the four frequencies  W j + 4 ((i xor j) mod (W/4)) + {0..3},  W = dh / 8.
__host__ __device__ __forceinline__ int lane_freq(int dh, int i, int j, int e) {
  const int W = dh / 8, nch = W / 4;
  return W * j + 4 * ((i ^ j) & (nch - 1)) + e;
}

// ---- work split ---------------------------------------------------------------------------
// largest u in [0, n) with pfx[u] <= x < pfx[u+1]  (x < pfx[n] assumed)
__device__ __forceinline__ int find_unit(const int32_t* pfx, int n, int64_t x) {
  int lo = 0, hi = n;  // invariant: pfx[lo] <= x < pfx[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if ((int64_t)pfx[mid] <= x)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// Two ways to deal T blocks to n CTAs.  By range: CTA c owns blocks [c T / n, (c + 1) T / n), whatever
// units they belong to; a CTA that meets a second unit pays a second prologue and merge (about
// kSegmentCost tiles of work).  By unit: unit u gets c_u = floor(nb_u n / T) CTAs (at least one) of equal
// shares, and nobody meets two units.  The second is taken when its largest share is within that
// cost of T / n: few units of similar size (2048 tokens x 8 heads: a step 22.3 -> 17.2 us, three rows of up
// to 6001 tokens x 8 heads 40.3 -> 33.1 us; by range half the CTAs met two units).  Call with a whole warp.
constexpr int kSegmentCost = 30;
struct UnitSplit {
  bool by_unit;
  int u, first, count;  // the unit `cta` works for, its first CTA, its CTAs
};
__device__ __forceinline__ UnitSplit split_by_unit(const int32_t* pfx, int n_units, int n_ctas, int tiles_per_block,
                                                   int cta) {
  UnitSplit r;
  r.by_unit = false; r.first = r.count = 0; r.u = 0;
  const uint32_t T = (uint32_t)pfx[n_units];
  if (n_units > n_ctas || T == 0 || T >= (1u << 24)) return r;
  const int lane = threadIdx.x & 31;
  const float per_block = (float)n_ctas / (float)T;
  const uint64_t bound = (uint64_t)T + (uint64_t)max(1, kSegmentCost / tiles_per_block) * n_ctas;
  auto blocks_of = [&](int i) { return i < n_units ? (uint32_t)(pfx[i + 1] - pfx[i]) : 0u; };
  auto ctas_of = [&](uint32_t nb) { return nb == 0 ? 0u : max(1u, min(nb, (uint32_t)((float)nb * per_block))); };
  uint32_t total = 0;
  bool fits = true;
  for (int base = 0; base < n_units; base += 32) {
    const uint32_t nb = blocks_of(base + lane), c = ctas_of(nb);
    total += c;
    fits = fits && (uint64_t)nb * n_ctas <= c * bound;  // share nb / c against T / n + cost
  }
  total = __reduce_add_sync(0xffffffffu, total);
  if (!__all_sync(0xffffffffu, fits) || total > (uint32_t)n_ctas) return r;
  r.by_unit = true;
  uint32_t carry = 0;
  for (int base = 0; base < n_units; base += 32) {
    const uint32_t c = ctas_of(blocks_of(base + lane));
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const uint32_t first = carry + x - c;
    const unsigned hit = __ballot_sync(0xffffffffu, (uint32_t)cta >= first && (uint32_t)cta < first + c);
    if (hit) {
      const int src = __ffs(hit) - 1;
      r.u = base + src;
      r.first = (int)__shfl_sync(0xffffffffu, first, src);
      r.count = (int)__shfl_sync(0xffffffffu, c, src);
      break;
    }
    carry += __shfl_sync(0xffffffffu, x, 31);
  }
  return r;
}
// first block of share i of n of a unit's nb
__device__ __forceinline__ int64_t share_start(int i, int n, int64_t nb) { return (int64_t)i * nb / n; }

// ---- K stage: what a tile needs of its page ---------------------------------------------------
// A 16-token page is staged whole; of a larger page the header + group scales, the slice of the theta
// bit stream of the tile's 16 tokens and the slice of their radius bytes go to fixed offsets; plus the
// tile's 16 positions.  Every piece keeps the phase inside 16 bytes that it has in the pool.
constexpr int kKHdr = 0;    // 8 header bytes + up to 8 scales = 40, + 12 phase
constexpr int kKTh = 64;    // 16 tokens x 8 groups x 6 bits = 96 bytes + 15 phase
constexpr int kKRd = 176;   // 16 tokens x 8 groups x 1 or 2 bytes + 15 phase
// int8 radii: stages of 384 bytes, positions in the last 64; f16: 512
static_assert(kKTh + 112 <= kKRd && kKRd + 128 + 16 <= 384 - 64 && kKRd + 256 + 16 <= 512 - 64, "K stage layout");
// the largest 16-token page, 8 + 32 + 96 + 128 (256) bytes + 12 phase, ends before the positions as well

// barriers of a team (8 bytes each, kBarStride per team)
enum { kBarKFull = 0, kBarKeys = kKStages, kBarKeys2, kBarLogits, kBarWeights, kBarV, kBarOut, kBarVote, kBarDrain, kBarCount };
static_assert(kBarCount * 8 <= kBarStride, "barrier block");

// A team of four warps rebuilds 128 keys (eight 16-token tiles) into tensor memory, its driver warp --
// which also fetches everything -- issues the two contractions:
//   teams    page bytes -> centroid rows x radius, rotated by the key's angle, bf16 hi | lo -> TMEM
//   driver   logits[128 tokens x 16] = keys . query   (A from TMEM; columns hi | lo of the query heads)
//   teams    thread = token row: softmax weights -> shared memory
//   driver   out[dh x 16] += V^T weights              (A = the V tiles as TMA wrote them, transposed)
// The accumulators of both contractions stay in TMEM, so a team thread holds one pass's cos/sin and the
// keys in flight and nothing else, twelve team warps fit an SM (the mma.sync version it replaced: eight, at
// 244 registers, and shuffles, ldmatrix and accumulator moves around both products).
// Bound: instruction issue and the waits between the roles, not HBM.  A 96-bit, 32768-token, batch-8 layer
// step, merge included, in a short loop: 159 -> 141 us (3.4 -> 3.8 TB/s of the bytes it has to read): 670
// instructions a tile instead of 755, since team addresses lie at constant offsets and stay in registers (147), then
// cos/sin past L1.
// Lane map of the rebuild (lane = 4 r + j): rows r and r + 8 of a tile are the lane's two tokens; in each
// rotary half the lane owns the contiguous block of W = dh / 8 dimensions  W j .. W j + W - 1, and in the
// other half the same block shifted by dh / 2: the RoPE partner of every value a lane holds is in the same
// lane, and for g = 16, dh = 128 a lane needs two centroid indices and two radii per token.
// PACK (<= 4 query heads per KV head): query and weight columns are [hi 0..3 | lo 0..3 | 0], else
// [hi 0..7 | lo 0..7].
// MODE bit 0 clear: 16-token pages with int8 radii (the serving configuration: page size and
// radius format are compile-time constants and the page image is staged word for word); set: any
// page size / radius format.  MODE bit 1: the logits / per-tile statistics side outputs.
template <int DH, typename VT, bool ROT, int MODE, bool PACK>
__global__ void __launch_bounds__(kDecodeThreads, 1) decode_splitk_kernel(const __grid_constant__ DecodeArgs a) {
  constexpr bool EXTRA = (MODE & 2) != 0, FAST = (MODE & 1) == 0;
  constexpr int W = DH / 8;     // dims a lane owns in each rotary half
  constexpr int NCH = W / 4;    // 16-byte chunks of those dims
  constexpr int V_TILE = 16 * DH * 2;
  constexpr int HEADS = PACK ? 4 : 8;
  constexpr bool kBf16 = std::is_same<VT, __nv_bfloat16>::value;
  // instruction descriptors: fp32 accumulate, 128 x 16; keys and query are bf16, weights and V of V's type
  constexpr uint32_t kIdescShape = (1u << 4) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
  constexpr uint32_t kIdescQK = kIdescShape | (1u << 7) | (1u << 10);
  constexpr uint32_t kIdescPV = kIdescShape | (kBf16 ? (1u << 7) | (1u << 10) : 0u) | (1u << 15) | (1u << 16);

  extern __shared__ __align__(1024) uint8_t smem[];
  const sphkv_decode_params& p = a.p;
  // What the loops use most of the thread's place comes out of shuffles, whose results stay in registers: short of those,
  // the compiler reads the special register again, and waits for it, or makes an address again at every use.  Of four such
  // addresses two fit beside the code for 16-token int8 pages, or beside dh 64 (barriers or the base of shared memory as
  // well: spills, 8 x 32768 147 -> 159 us); elsewhere the team alone (2 x 30614 tokens, 32-token pages: 55.6 us with
  // none, 57.0 with the two, 54.8).
  constexpr bool kKeepBases = FAST || DH == 64;
  auto keep = [](bool yes, auto x) { return yes ? __shfl_sync(0xffffffffu, x, 0) : x; };
  const int warp = keep(true, (int)(threadIdx.x >> 5));
  const int lane = __shfl_sync(0xffffffffu, (int)(threadIdx.x & 31), (int)(threadIdx.x & 31));
  const bool driver = warp >= 4 * kTeams;
  const int team = keep(!kKeepBases, driver ? warp - 4 * kTeams : warp >> 2);
  const bool in_use = team < a.teams;  // (the fourth driver warp never is; idle warps do not use their addresses)

  const uint32_t smem0 = smem_u32(smem);
  const uint32_t q_u32 = smem0;
  const uint32_t bar = smem0 + smem_q_bytes(DH) + team * kSmemTeamBars;
  const uint32_t votes = bar + kBarStride;   // [2][4 warps]
  const uint32_t wmax = votes + 32;          // [4 warps][8 heads]
  // of a team: [4 warps][8 heads] (sum, true maximum), [8 heads] reference maximum
  auto stats_of = [&](int t) { return reinterpret_cast<float*>(smem + smem_head_bytes(DH) + a.teams * smem_team_bytes(DH) + t * kSmemStats); };
  auto mref_of = [&](int t) { return reinterpret_cast<float*>(smem + smem_q_bytes(DH) + t * kSmemTeamBars + kBarStride + 32 + 128); };
  volatile uint32_t* shared_words = reinterpret_cast<volatile uint32_t*>(smem + smem_q_bytes(DH) + kTeams * kSmemTeamBars);
  const uint32_t v_buf = keep(kKeepBases, smem0 + smem_head_bytes(DH) + team * smem_team_bytes(DH));
  const uint32_t p_buf = v_buf + smem_v_bytes(DH), k_ring = p_buf + kSmemP, meta = k_ring + kSmemK;
  const uint32_t cb_off = smem_fixed_bytes(DH, a.teams);

  // ---- set-up: barriers, tensor memory, the zero columns of the weights and of the query operand ----
  if (driver && in_use && lane == 0) {
    for (int i = 0; i < kKStages; ++i) mbar_init(bar + 8 * (kBarKFull + i), 33);  // 32 copy arrivals + plain stores
    mbar_init(bar + 8 * kBarKeys, 4);
    mbar_init(bar + 8 * kBarKeys2, 4);
    mbar_init(bar + 8 * kBarLogits, 1);
    mbar_init(bar + 8 * kBarWeights, 4);
    mbar_init(bar + 8 * kBarV, 1);
    mbar_init(bar + 8 * kBarOut, 1);
    mbar_init(bar + 8 * kBarVote, 4);
    mbar_init(bar + 8 * kBarDrain, 1);
  }
  if (!driver) {
    if (in_use)
      for (int i = threadIdx.x & 127; i < kSmemP / 16; i += 128) sts128(p_buf + 16 * i, 0, 0, 0, 0);
    for (int i = threadIdx.x; i < smem_q_bytes(DH) / 16; i += kTeamThreads) sts128(q_u32 + 16 * i, 0, 0, 0, 0);
  }
  if (warp == 4 * kTeams + 3) {
    if (lane == 0) shared_words[1] = 0;
    tmem_alloc(smem_u32(const_cast<uint32_t*>(shared_words)), kTmemCols);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, shared_words[0], 0);
  const uint32_t tmem = keep(kKeepBases, tmem_base + team * kTeamCols);
  // everything above touched shared and tensor memory only: this grid's launch overlaps the tail of the
  // kernel before it in the stream (the previous step's merge kernel, which lets it in early)
  griddep_wait();
  bool dead = false;  // a bounded wait ran out: stop working, keep meeting the barriers

  // ---- block prefix per unit: computed by warp 0 of every CTA, or read from the plan kernel's output
  //      when there are many units ----
  const int32_t* pfx = a.pfx;
  if (a.plan_in_kernel) {
    int32_t* pfx_s = reinterpret_cast<int32_t*>(smem + cb_off + a.cb_smem_bytes);
    if (warp == 0) {
      int carry = 0;
      for (int base = 0; base < a.n_units; base += 128) {
        int v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // four loads in flight
          const int i = base + 32 * q + lane;
          v[q] = i < a.n_units ? p.num_blocks[(i % p.B) * p.Hkv + i / p.B] : 0;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = base + 32 * q + lane;
          if (base + 32 * q >= a.n_units) break;
          v[q] = v[q] < 0 ? 0 : (v[q] > p.max_blocks ? p.max_blocks : v[q]);
          int x = v[q];
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
          }
          if (i < a.n_units) pfx_s[i] = carry + x - v[q];
          carry += __shfl_sync(0xffffffffu, x, 31);
        }
      }
      if (lane == 0) pfx_s[a.n_units] = carry;
    }
    __syncthreads();
    pfx = pfx_s;
  }
  const int64_t T = pfx[a.n_units];
  const int N = FAST ? 16 : p.page_size;
  int64_t start, end;
  int u, unit_ctas = 0;  // unit_ctas: CTAs of the one unit of this CTA; 0: dealt by range
  const int n_ctas = (int)min((int64_t)a.n_ctas, T);  // every CTA below has a block
  {
    const UnitSplit us = split_by_unit(pfx, a.n_units, n_ctas, N >> 4, blockIdx.x);
    if (us.by_unit) {
      unit_ctas = us.count;
      u = us.u;
      const int64_t first = pfx[u], nb = (int64_t)pfx[u + 1] - first;
      start = end = first;
      if (us.count > 0) {  // else: a CTA that no unit needs
        start = first + share_start(blockIdx.x - us.first, us.count, nb);
        end = first + share_start(blockIdx.x - us.first + 1, us.count, nb);
      }
    } else {
      start = end = 0;
      if ((int)blockIdx.x < n_ctas) {
        start = cta_range_start(blockIdx.x, n_ctas, T);
        end = cta_range_start(blockIdx.x + 1, n_ctas, T);
      }
      u = start < end ? find_unit(pfx, a.n_units, start) : 0;
    }
  }

  const int TPP = N >> 4;  // 16-token tiles per page: 1, 2, 4 or 8
  const int tpp_shift = 31 - __clz(TPP);
  const int fmt = FAST ? SPHKV_RADIUS_I8 : p.radius_fmt;
  const uint32_t rb = fmt == SPHKV_RADIUS_F16 ? 2u : 1u;
  const uint32_t kst_bytes = rb == 2 ? 512 : 384, kst_pos = kst_bytes - 64;  // K stage of a tile, its positions
  const int n_stages = rb == 2 ? 2 : kKStages;
  // per tier slot: b_theta | log2(g) << 8 | duplicated << 12 | codebook offset in shared
  // memory << 13, held by lanes 0..3 and read with a shuffle
  uint32_t tier_word = 0;
  if (lane < SPHKV_MAX_TIER_SLOTS && lane < p.tiers.n_slots) {
    int g_l = 16, b_l = 1, off_l = 0, dup_l = 0;
#pragma unroll
    for (int s = 0; s < SPHKV_MAX_TIER_SLOTS; ++s)
      if (s == lane) { g_l = p.tiers.g[s]; b_l = p.tiers.bits[s]; off_l = a.cb_smem_off[s]; dup_l = a.cb_dup[s]; }
    tier_word = (uint32_t)b_l | ((uint32_t)(g_l == 32 ? 5 : 4) << 8) | ((uint32_t)dup_l << 12) |
                ((uint32_t)off_l << 13);
  }
  auto tier_of = [&](int slot) { return __shfl_sync(0xffffffffu, tier_word, slot); };

  // ---- the CTA's block range, one segment per unit it meets.  Units are walked KV head major
  //      (u = hkv * B + b) so that neighbouring segments share their codebooks; tables are indexed by the
  //      external unit id b * Hkv + hkv.  Macro tile k of a team = tiles [(k * teams + team) * width,
  //      + width): the teams walk a segment together (its tiers change the work per tile) and a short
  //      segment is spread over all of them. ----
  int hkv = 0, b = 0, lb0 = 0, seg_tiles = 0, width = 1, rounds = 0;
  int64_t seg_end = start;
  auto first_tile = [&](int k) { return (k * a.teams + team) * width; };
  auto next_segment = [&]() {
    while ((int64_t)pfx[u + 1] <= start) ++u;  // skip units without blocks
    seg_end = end < (int64_t)pfx[u + 1] ? end : (int64_t)pfx[u + 1];
    lb0 = (int)(start - pfx[u]);
    seg_tiles = (int)(seg_end - start) * TPP;
    hkv = u / p.B;
    b = u - hkv * p.B;
    const int per_round = kMacroTiles * a.teams;
    const int all_rounds = (seg_tiles + per_round - 1) / per_round;
    width = (seg_tiles + all_rounds * a.teams - 1) / (all_rounds * a.teams);
    rounds = !in_use || dead || first_tile(0) >= seg_tiles ? 0 : (first_tile(all_rounds - 1) < seg_tiles ? all_rounds : all_rounds - 1);
  };
  auto give_up = [&]() {  // a wait was not answered within its bound: the host sees the status bit
    if (lane == 0) {
      if (p.status) atomicOr(p.status, SPHKV_ST_TIMEOUT);
      shared_words[1] = 1;
    }
  };

  // The two roles share no code from here on (each is compiled for its own number of registers) and meet
  // at the team barriers only: a driver fetches the first macro tiles of the next segment while the
  // teams merge the last one.
  if (driver) {
  regs_down<kDriverRegs>();
  uint32_t par_keys = 0, par_weights = 0, par_v = 0, par_out = 0;
  const uint64_t v_policy = policy_evict_first();  // V is read once per step, the cos/sin rows many times
  for (; start < end; start = seg_end, ++u) {
    next_segment();
    const int u_ext = b * p.Hkv + hkv;
    // the CTA of a unit's first block tells the merge kernel which CTAs the unit has (by range: the last one
    // is the largest c with c T / n < the unit's end)
    if (warp == 4 * kTeams + 3 && lane == 0 && lb0 == 0) {
      const int count = unit_ctas > 0 ? unit_ctas : (int)(((int64_t)pfx[u + 1] * n_ctas - 1) / T) - (int)blockIdx.x + 1;
      a.spans[u] = (uint32_t)blockIdx.x | ((uint32_t)count << 16);
    }
    // ---- block table -> pointer table of 32 tiles at a time (lane = tile), the dependent loads in separate
    //      rounds so that no round waits for a load it issued itself.  How many tokens the page can hold
    //      follows from the size of its theta stream; the header's count is applied by the teams, from
    //      the staged bytes (reading it here would be one more memory latency before the page copies) ----
    const int32_t* bt_row = p.block_table + (int64_t)u_ext * p.max_blocks;
    const int32_t* st_row = p.bits_table + (int64_t)u_ext * p.max_blocks;
    int mf_phys = -2, mf_slot = 0, mf_poff = 0, mf_toff = 0, mf_roff = 0;
    auto meta_blocks = [&](int kb) {
      const int kk = kb + (lane >> 3), x = lane & 7, t = first_tile(kk) + x;
      mf_phys = -2; mf_slot = 0; mf_poff = mf_toff = mf_roff = 0;  // -2: no such tile
      if (kk < rounds && x < width && t < seg_tiles) {
        const int lb = lb0 + (t >> tpp_shift);
        mf_phys = bt_row[lb];
        mf_slot = st_row[lb];
        if (mf_phys < 0) mf_phys = -1;  // a hole in the block list
      }
    };
    auto meta_pointers = [&]() {
      if (mf_phys < 0) { mf_slot = 0; return; }
      if (mf_phys >= p.n_pages) {
        if (p.status) atomicOr(p.status, SPHKV_ST_BAD_BLOCK);
        mf_phys = -1;
      }
      if (mf_slot < 0 || mf_slot >= p.tiers.n_slots) {
        if (p.status) atomicOr(p.status, SPHKV_ST_BAD_SLOT);
        mf_phys = -1;
        mf_slot = 0;
      }
      if (mf_phys < 0) return;
      mf_poff = p.ptable[3 * (int64_t)mf_phys + 0];
      mf_toff = p.ptable[3 * (int64_t)mf_phys + 1];
      mf_roff = p.ptable[3 * (int64_t)mf_phys + 2];
    };
    auto meta_store = [&](int kb) {
      TileMeta m;
      m.phys = mf_phys; m.poff = mf_poff; m.where = m.rad = 0;
      if (mf_phys >= 0) {
        const int sub = (first_tile(kb + (lane >> 3)) + (lane & 7)) & (TPP - 1);
        const uint32_t bits = p.tiers.bits[mf_slot], G = DH / p.tiers.g[mf_slot];
        const uint32_t phase = (uint32_t)mf_poff & 15u;
        const int th_bytes = mf_roff - mf_toff;
        uint32_t th, rd;
        if (TPP == 1) {
          th = phase + (uint32_t)(mf_toff - mf_poff);
          rd = phase + (uint32_t)(mf_roff - mf_poff);
        } else {
          th = kKTh + (((uint32_t)mf_toff + ((16u * sub * G * bits) >> 3)) & 15u);
          rd = kKRd + (((uint32_t)mf_roff + 16u * sub * G * rb) & 15u);
        }
        // Sections may be padded: 16-token pages are staged whole and have to fit, of larger ones each section is
        // found by itself.  With int8 radii 16-token pages start their theta stream right behind the scales.
        const int lead = mf_toff - mf_poff;
        const bool fits = TPP == 1 ? rd + 16 * G * rb <= kst_pos && rd < 512 : lead < 1024 && th_bytes < 65536;
        if ((FAST ? lead != (int)(8 + 4 * G) : lead < (int)(8 + 4 * G)) || th_bytes < 0 || !fits) {
          // the pointer table disagrees with the page format: not a page this kernel can read
          if (p.status) atomicOr(p.status, SPHKV_ST_BAD_BLOCK);
          m.phys = -1;
        } else {
          int count = min(N, (int)((uint32_t)th_bytes * 8u / (G * bits)));
          if (G * bits < 8 || (int)(((uint32_t)count * G * bits + 7) >> 3) != th_bytes)
            // several counts share a stream size, or the stream is padded: the header it is
            count = min(count, (int)p.k_pages[mf_poff + 1]);
          const int tokens = min(16, max(0, count - 16 * sub));
          m.where = (uint32_t)tokens | ((uint32_t)mf_slot << 8) | (phase << 12) | (th << 16) | ((uint32_t)sub << 28);
          m.rad = rd | ((uint32_t)(lead & 0x7F) << 9) | ((uint32_t)th_bytes << 16);
          if (!FAST) m.where |= (uint32_t)(lead >> 7) << 25;  // read for pages of more than one tile only
        }
      }
      sts_meta(meta + ((kb * kMacroTiles + lane) & (kMetaRing - 1)) * 16, m);
      __syncwarp();
    };
    auto get_meta = [&](int k, int x) { return lds_meta(meta + ((k * kMacroTiles + x) & (kMetaRing - 1)) * 16); };

    // V tiles of macro tile k: one box of dh / 64 x 16 rows x 128 bytes per tile through the tensor map,
    // hardware swizzle = chunk ^ (row & 7).  Returns the tiles that hold tokens.
    auto issue_v = [&](int k) -> unsigned {
      TileMeta m;
      m.phys = -2; m.where = 0;
      if (lane < width) m = get_meta(k, lane);
      const bool have = meta_tokens(m) > 0;
      const unsigned mask = __ballot_sync(0xffffffffu, have);
      if (lane == 0) {
        if (mask)
          mbar_expect_tx(bar + 8 * kBarV, __popc(mask) * V_TILE);
        else
          mbar_arrive(bar + 8 * kBarV);
      }
      __syncwarp();
      if (have) {
        const int y = m.phys * N + 16 * meta_sub(m);
        tma_load_3d(v_buf + lane * V_TILE, &a.v_map, 0, y, 0, bar + 8 * kBarV, v_policy);
      }
      return mask;
    };

    // K stage of macro tile k, four lanes per tile.  A piece of the pool travels as the 16-byte chunks that
    // hold it (it keeps its byte phase inside the first), its last, partial chunk as words: nothing past
    // the piece's last word is read.  16-token pages are one piece; of larger ones the header, the
    // tile's slice of the theta stream and of the radii.  Pools off a 16-byte boundary: words only.
    auto issue_k = [&](int k, int stage) {
      const int x = lane >> 2, q = lane & 3;
      TileMeta m;
      m.phys = -2; m.poff = 0; m.where = 0; m.rad = 0;
      if (x < width) m = get_meta(k, x);
      const uint32_t tw = tier_of(meta_slot(m));
      const uint32_t kb = k_ring + (stage * kMacroTiles + x) * kst_bytes;
      auto piece = [&](uint32_t dst, uint32_t src, uint32_t stop) {
        const uint32_t s0 = src & ~15u;
        uint32_t o = src & ~3u;
        if (a.wide) {
          const uint32_t full = max(stop & ~15u, s0);
          for (o = s0 + 16 * q; o < full; o += 64) cp_async_16(dst + (o - s0), p.k_pages + o);
          o = full;
        }
        for (o += 4 * q; o < stop; o += 16) cp_async_4(dst + (o - s0), p.k_pages + o);
      };
      if (m.phys >= 0) {
        const uint32_t bits = tw & 0xFF, G = (uint32_t)DH >> ((tw >> 8) & 0xF);
        const uint32_t poff = (uint32_t)m.poff;
        const int sub = meta_sub(m);
        const uint32_t stop = poff - meta_hdr(m) + meta_radius(m) + (uint32_t)meta_tokens(m) * G * rb;
        if (FAST && a.wide) {  // at most 20 chunks, then the last words
          const uint32_t s0 = poff & ~15u, full = stop & ~15u;
#pragma unroll
          for (int e = 0; e < 20; e += 4)
            if (s0 + 16 * (q + e) < full) cp_async_16(kb + 16 * (q + e), p.k_pages + s0 + 16 * (q + e));
          if (full + 4 * q < stop) cp_async_4(kb + (full - s0) + 4 * q, p.k_pages + full + 4 * q);
        } else if (TPP == 1) {
          piece(kb, poff, stop);
        } else {
          const uint32_t t0 = 16u * sub, t1 = t0 + (uint32_t)meta_tokens(m);
          const uint32_t toff = poff + (((m.rad >> 9) & 0x7F) | (((m.where >> 25) & 0x7) << 7)), roff = toff + (m.rad >> 16);
          piece(kb + kKHdr, poff, poff + 8 + 4 * G);
          piece(kb + kKTh, toff + ((t0 * G * bits) >> 3), toff + ((t1 * G * bits + 7) >> 3));
          piece(kb + kKRd, roff + t0 * G * rb, roff + t1 * G * rb);
        }
        if (ROT) {
          const int32_t* ps = p.positions + ((uint32_t)m.phys * (uint32_t)N + 16u * sub + 4 * q);
          if (a.wide) {
            cp_async_16(kb + kst_pos + 16 * q, ps);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) cp_async_4(kb + kst_pos + 16 * q + 4 * e, ps + e);
          }
        }
      } else if (ROT && x < width) {
        sts128(kb + kst_pos + 16 * q, ~0u, ~0u, ~0u, ~0u);  // no page: its positions read as "no token"
      }
      cp_async_arrive(bar + 8 * (kBarKFull + stage));
      __syncwarp();
      if (lane == 0) mbar_arrive(bar + 8 * (kBarKFull + stage));
    };

    unsigned v_tiles = 0;
    if (rounds > 0) {
      meta_blocks(0);
      meta_pointers();
      meta_store(0);
      for (int i = 0; i < min(rounds, n_stages); ++i) issue_k(i, i);
      v_tiles = issue_v(0);
      meta_blocks(4);
    }
    int lost = 0;  // a wait ran out: 1 with V tiles on their way, 2 without
    bool started = false;
    const uint64_t q_desc = smem_desc(q_u32, 128, 256, 0), p_desc = smem_desc(p_buf, 128, 256, 0);
    const uint64_t v_desc = smem_desc(v_buf, DH == 128 ? 2048 : 0, 1024, 2);
    for (int k = 0, st = 0; k < rounds; ++k) {
      // the metadata of the next four macro tiles, stored before the first of them is fetched (k + 3 at most)
      // and after the teams have finished what it replaces in the ring (k - 5 and before)
      if ((k & 3) == 0)
        meta_pointers();
      else if ((k & 3) == 1)
        meta_store(k + 3);
      else if ((k & 3) == 3)
        meta_blocks(k + 5);
      // the first chunks of the keys are multiplied while the teams rebuild the last
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        if (!__all_sync(0xffffffffu, mbar_wait(bar + 8 * (kBarKeys + part), par_keys))) { lost = 1; break; }
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int c = 2 * NCH * part; c < 2 * NCH * (part + 1); ++c)  // per chunk: hi, hi, lo, lo of the two rotary halves
            mma_ts(tmem + kColLogits, tmem + kColKeys + 8 * c, q_desc + (uint64_t)((((c & 1) * NCH + (c >> 2)) * 512) >> 4), kIdescQK, c > 0);
          if (part == 1) mma_commit(bar + 8 * kBarLogits);
        }
      }
      if (lost) break;
      par_keys ^= 1;
      __syncwarp();
      if (k + n_stages < rounds) issue_k(k + n_stages, st);  // the team has read macro tile k's stage
      if (++st == n_stages) st = 0;
      const bool got = mbar_wait(bar + 8 * kBarWeights, par_weights) && mbar_wait(bar + 8 * kBarV, par_v);
      if (!__all_sync(0xffffffffu, got)) { lost = 1; break; }
      par_weights ^= 1;
      par_v ^= 1;
      tc_fence_after();
      if (elect_one()) {
        // A = V^T: 64-dim halves 2048 bytes apart (dh 64: the second half repeats the first, its rows of
        // the accumulator are not read), 8-token groups 1024 apart
#pragma unroll
        for (int x = 0; x < kMacroTiles; ++x)
          if ((v_tiles >> x) & 1)
            mma_ss(tmem + kColOut, v_desc + (uint64_t)((x * V_TILE) >> 4), p_desc + (uint64_t)((x * 512) >> 4), kIdescPV,
                   started || (v_tiles & ((1u << x) - 1u)) != 0);
        mma_commit(bar + 8 * kBarOut);
      }
      started = started || v_tiles != 0;
      __syncwarp();
      if (!__all_sync(0xffffffffu, mbar_wait(bar + 8 * kBarOut, par_out))) { lost = 2; break; }
      par_out ^= 1;
      if (k + 1 < rounds) v_tiles = issue_v(k + 1);
    }
    if (lost) {
      // Nothing that this driver started may still write when the CTA's memory is given back: page bytes, V tiles
      // and products are awaited, each within the same bound.  Reached once at most: it has no rounds in later
      // segments.
      dead = true;
      give_up();
      cp_async_wait_all();
      if (lost == 1) (void)mbar_wait(bar + 8 * kBarV, par_v);
      __syncwarp();
      if (elect_one()) mma_commit(bar + 8 * kBarDrain);
      __syncwarp();
      (void)mbar_wait(bar + 8 * kBarDrain, 0);
    }
    dead = dead || shared_words[1] != 0;
  }
  } else {
  regs_up<kTeamRegs>();
  int cb_head_loaded = -1;
  auto stage_codebooks = [&]() {
    if (hkv == cb_head_loaded) return;
    const sphkv_tiers& tg = p.tiers;
    for (int s = 0; s < tg.n_slots; ++s) {
      // [group][centroid][g floats]; a duplicated slot (g = 16) keeps two copies of every 64-byte row
      // in one 128-byte slot, the second for odd token rows.  Group number gh of a rotary half is shifted
      // by 16 gh bytes: the four lanes of a token, reading stored chunk i of their rows together, never
      // meet in a bank.  The chunks of the W dims that quad member j reads are stored XOR-ed with j, the
      // order of the cos/sin table, so a lane's address is its row plus a constant.
      const int g = tg.g[s], bits = tg.bits[s], G = DH / g, cpr = g >> 2;
      const int dup = a.cb_dup[s];
      const float* src = p.codebooks + ((int64_t)(hkv * tg.n_slots + s) * tg.G_max) * tg.C_max * tg.g_max;
      const uint32_t dst = smem0 + cb_off + a.cb_smem_off[s];
      const int lc = g == 32 ? 3 : 2;  // log2 of the chunks per row
      const int chunks = (G << bits) << lc;
      // asynchronous 16-byte copies: every chunk of the codebook is in flight at once instead
      // of one load-store round trip per loop iteration (the caller waits for the group)
      for (int i = threadIdx.x; i < chunks; i += kTeamThreads) {
        const int c4 = i & (cpr - 1), row = i >> lc;
        const int c = row & ((1 << bits) - 1), gam = row >> bits;
        const int to = c4 ^ ((((gam * g + c4 * 4) & (DH / 2 - 1)) / W) & (NCH - 1));
        const int gh = gam >= (G >> 1) ? gam - (G >> 1) : gam;
        const uint32_t at = dst + gh * 16 + (gam >= (G >> 1) ? 64 : 0);
        const float4* sp = reinterpret_cast<const float4*>(src + (gam * tg.C_max + c) * tg.g_max) + c4;
        if (dup) {
          cp_async_16(at + (row * 8 + to) * 16, sp);
          cp_async_16(at + (row * 8 + 4 + to) * 16, sp);
        } else {
          cp_async_16(at + (row * cpr + to) * 16, sp);
        }
      }
    }
    cb_head_loaded = hkv;
  };
  // Query operand of a unit: bf16 hi (truncated) and lo parts of q * sm_scale * log2(e), 16 columns x 16
  // dims per block, K-major, no swizzle: 8-column groups at 256 bytes, 8-dim groups at 128.  Block
  // half * NCH + i holds, for lane quad member j, the four dims of chunk i: k = 4 j + e.  A thread loads its
  // (at most three) values at once, before the codebooks, and stores both parts of each after them.
  constexpr int kQLoads = (HEADS * DH + kTeamThreads - 1) / kTeamThreads;
  float q_val[kQLoads];
  auto load_query = [&]() {
    const int64_t q0 = ((int64_t)b * p.Hq + (int64_t)hkv * a.grp) * DH;
#pragma unroll
    for (int l = 0; l < kQLoads; ++l) {
      const int i = threadIdx.x + l * kTeamThreads;
      q_val[l] = i < a.grp * DH ? load_as_float(p.q, p.q_dtype, q0 + i) : 0.f;
    }
  };
  auto stage_query = [&]() {
    const float qscale = p.sm_scale * kLog2e;
#pragma unroll
    for (int l = 0; l < kQLoads; ++l) {
      const int i = threadIdx.x + l * kTeamThreads;
      if (i >= a.grp * DH) break;
      const int head = i / DH, d = i % DH, half = d / (DH / 2), f = d % (DH / 2);
      const int j = f / W, chunk = ((f % W) >> 2) ^ (j & (NCH - 1)), k = 4 * j + (f & 3);
      const float x = q_val[l] * qscale;
      const float hi = __uint_as_float(__float_as_uint(x) & 0xFFFF0000u);
      auto put = [&](int n, float v) {
        reinterpret_cast<__nv_bfloat16*>(smem + (half * NCH + chunk) * 512 + (n >> 3) * 256 +
                                         (k >> 3) * 128)[(n & 7) * 8 + (k & 7)] = __float2bfloat16_rn(v);
      };
      put(head, hi);  // exact
      put(head + HEADS, x - hi);
    }
  };
  uint32_t par_k = 0, par_logits = 0, par_out = 0, par_vote = 0;
  for (; start < end; start = seg_end, ++u) {
    next_segment();
    const int64_t ml_head = (int64_t)p.max_blocks * TPP * 2;
    load_query();
    stage_codebooks();
    cp_async_commit();
    stage_query();
    cp_async_wait<0>();  // this thread's codebook copies; the barrier publishes everyone's
    fence_async_smem();  // and the query operand to the tensor core
    teams_barrier();

    // online-softmax state of the team, identical in its 128 threads: the reference maximum of every head
    // (it follows the true one within 2^kSlack, so that accumulator and sums are rarely rescaled); per
    // thread the sums and true maxima of its own token rows
    constexpr float kSlack = 8.f;
    float m_ref[HEADS], m_true[HEADS], l_run[HEADS];
#pragma unroll
    for (int h = 0; h < HEADS; ++h) { m_ref[h] = m_true[h] = -INFINITY; l_run[h] = 0.f; }

    if (rounds > 0) {
      const int w = warp & 3;  // TMEM lanes 32 w .. 32 w + 31
      const int r = lane >> 2, j = lane & 3;
      const uint32_t tmem_rows = tmem + ((uint32_t)(32 * w) << 16);

      // lane constants of the tier slot of the current tile, recomputed only when the slot changes
      // (block lists keep the pages of a tier together)
      int c_slot = -1;
      uint32_t c_bits = 1, c_mask = 1, c_rowb = 64, c_cb_lo = 0, c_cb_hi = 0;
      // bit offset of the centroid index of (token r, first half) and byte offset of its radius: relative to
      // the tile's theta / radius slice, or (FAST) to the page start and to the first radius byte; steps to
      // token r + 8 and to the group of the second half
      uint32_t c_bit0 = 0, c_tok = 0, c_half = 0, c_rad0 = 0, c_rtok = 0, c_rhalf = 0;
      uint32_t c_sc[2] = {0, 0};  // byte offset of its group's scale in the header piece
      auto load_slot_constants = [&](int slot) {
        const uint32_t tw = tier_of(slot);
        const int lg = (tw >> 8) & 0xF;
        const int G = DH >> lg;
        const int glo = (W * j) >> lg, ghi = glo + (G >> 1);
        const int sub_off = (W * j) & ((1 << lg) - 1);
        const int dup = (tw >> 12) & 1;
        c_bits = tw & 0xFF;
        c_mask = (1u << c_bits) - 1u;
        c_rowb = 4u << (lg + dup);  // bytes from one centroid row to the next
        const uint32_t base = smem0 + cb_off + (tw >> 13) + sub_off * 4 + (dup ? (r & 1) * 64 : 0);
        c_cb_lo = base + ((uint32_t)glo << c_bits) * c_rowb + 16 * glo;
        c_cb_hi = base + ((uint32_t)ghi << c_bits) * c_rowb + 16 * glo + 64;
        // 16-token pages: the theta stream starts 8 + 4 G bytes into the page (pagebuilder.py:8-33;
        // checked against the pointer table when the tile metadata is fetched)
        c_bit0 = (uint32_t)(r * G + glo) * c_bits + (FAST ? (8 + 4 * G) * 8 : 0);
        c_tok = 8u * G * c_bits;
        c_half = (uint32_t)(G >> 1) * c_bits;
        c_rad0 = (uint32_t)(r * G + glo) * rb;
        c_rtok = 8u * G * rb;
        c_rhalf = (uint32_t)(G >> 1) * rb;
        c_sc[0] = 8 + 4 * glo;
        c_sc[1] = 8 + 4 * ghi;
        c_slot = slot;
      };
      // table row of a key position: "no token" (-1) and out-of-range positions read row 0 (the softmax
      // raises the status bit of the latter)
      auto clamp_pos = [&](int pos) -> uint32_t { return (uint32_t)pos < (uint32_t)p.max_pos ? (uint32_t)pos : 0u; };
      // cos/sin of this lane's two key positions: one 256-bit load per (token, chunk) brings the
      // chunk's {cos x 4, sin x 4} (the table is L2 resident), issued for the next pass once this one
      // has used its own.  A row's lines are used whole by one load and not again: past the 30 KB of L1 that the
      // shared memory leaves (1 x 131072 88.5 -> 83.7 us, 8 x 32768 146.9 -> 141.0; the read-only path, without L1,
      // 84.4 and 143.8).  The other page formats still take the read-only path.  At 128 dims it costs them up to 4 %
      // of a long context (read-only / past L1, 1 x 131072: 16-token f16 radii 115.1 / 111.1, 32-token pages 112.7 / 110.6,
      // 128-token 110.5 / 107.7, with f16 radii 125.2 / 120.0; 8 x 32768: 162.6 / 160.1, 190.1 / 189.2, 187.2 / 186.5,
      // 194.0 / 193.8), nothing at 64 dims (within 0.3 %) nor of a short one (424 tokens: 14.25 / 14.39)
      float4 cs[2][NCH][2];
      const float4* cs_src[2] = {nullptr, nullptr};  // this lane's pieces of the two table rows
      auto cs_rows = [&](uint32_t st) {              // positions of K stage `st`
        if constexpr (ROT) {
#pragma unroll
          for (int tk = 0; tk < 2; ++tk)
            cs_src[tk] = reinterpret_cast<const float4*>(p.rope_table) +
                         (clamp_pos((int)lds32(st + kst_pos + 4 * r + 32 * tk)) * (DH / 4) + j * 2);
        }
      };
      auto issue_cs_chunk = [&](int i) {
        if constexpr (ROT) {
#pragma unroll
          for (int tk = 0; tk < 2; ++tk) {
            float4 &c = cs[tk][i][0], &n = cs[tk][i][1];
            if (FAST)
              asm volatile("ld.global.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                           : "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w), "=f"(n.x), "=f"(n.y), "=f"(n.z), "=f"(n.w)
                           : "l"(cs_src[tk] + i * 8));
            else
              asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                           : "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w), "=f"(n.x), "=f"(n.y), "=f"(n.z), "=f"(n.w)
                           : "l"(cs_src[tk] + i * 8));
          }
        }
      };
      // K stage of tile x in ring slot `slot`; parities of the slots are bits of par_k
      auto stage_at = [&](int slot, int x) { return k_ring + (slot * kMacroTiles + x) * kst_bytes; };
      auto meta_of = [&](int k, int x) { return lds_meta(meta + ((k * kMacroTiles + x) & (kMetaRing - 1)) * 16); };
      auto wait_k = [&](int slot) -> bool {
        const uint32_t par = (par_k >> slot) & 1u;
        par_k ^= 1u << slot;
        return __all_sync(0xffffffffu, mbar_wait(bar + 8 * (kBarKFull + slot), par));
      };
      // Centroid rows (shared-memory addresses) and radii of this lane's tokens r, r + 8 in the tiles of
      // both passes, [pass][2 token + half]; taken from the page bytes while the tensor core multiplies
      // the macro tile before
      uint32_t row[2][4];
      float rad[2][4];
      bool have[2];
      auto extract = [&](int k, int slot) {
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
          const int x = w + 4 * pass;
          TileMeta m;
          m.where = 0;
          if (x < width) m = meta_of(k, x);
          have[pass] = meta_tokens(m) != 0;
          if (!have[pass]) continue;
          if (meta_slot(m) != c_slot) load_slot_constants(meta_slot(m));
          const uint32_t kst = stage_at(slot, x);
          const uint32_t hd_ad = kst + meta_hdr(m), rd_ad = kst + meta_radius(m) + c_rad0;
          const uint32_t bit0 = 8 * (FAST ? meta_hdr(m) : meta_theta(m)) + c_bit0;
          float scl[2] = {1.f, 1.f};
          if (fmt != SPHKV_RADIUS_F16) {
            scl[0] = __uint_as_float(lds32(hd_ad + c_sc[0])) * (1.0f / 127.0f);
            scl[1] = __uint_as_float(lds32(hd_ad + c_sc[1])) * (1.0f / 127.0f);
          }
#pragma unroll
          for (int tk = 0; tk < 2; ++tk) {
            // the indices of both halves lie within (G / 2 + 1) b_theta <= 30 bits of the stream
            const uint32_t bit = bit0 + (tk ? c_tok : 0u), wa = kst + ((bit >> 5) << 2);
            const uint32_t both = __funnelshift_r(lds32(wa), lds32(wa + 4), bit);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              const uint32_t code = (hf ? both >> c_half : both) & c_mask;
              row[pass][2 * tk + hf] = (hf ? c_cb_hi : c_cb_lo) + code * c_rowb;
              const uint32_t ra = rd_ad + (tk ? c_rtok : 0u) + (hf ? c_rhalf : 0u);
              if (fmt == SPHKV_RADIUS_F16)
                rad[pass][2 * tk + hf] = __half2float(__ushort_as_half((unsigned short)(lds_u8(ra) | (lds_u8(ra + 1) << 8))));
              else
                rad[pass][2 * tk + hf] = scl[hf] * (float)lds_s8(ra);
            }
          }
        }
      };
      // this warp's stores to tensor memory are done: the driver may multiply them
      auto keys_ready = [&](int which) {
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar + 8 * which);
      };

      dead = !wait_k(0);
      if (!dead) {
        if (w < width) {
          cs_rows(stage_at(0, w));
#pragma unroll
          for (int i = 0; i < NCH; ++i) issue_cs_chunk(i);
        }
        extract(0, 0);
      }
      for (int k = 0, slot = 0, slot_n = 0; k < rounds && !dead; ++k, slot = slot_n) {
        slot_n = slot + 1 == n_stages ? 0 : slot + 1;  // the next macro tile's
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
          // the pass after this one: its positions decide the cos/sin rows fetched below
          bool more = w + 4 < width;
          uint32_t st_next = stage_at(slot, w + 4);
          if (pass == 1) {
            more = k + 1 < rounds && w < width;
            st_next = stage_at(slot_n, w);
            if (k + 1 < rounds && !wait_k(slot_n)) { dead = true; break; }
          }
          if (more) cs_rows(st_next);
          if (have[pass]) {
            // ---- rebuild and rotate the keys chunk by chunk; bf16 hi | lo parts to tensor memory ----
            // Operand split: hi = the upper 16 bits of the fp32 value (a bf16 number, by truncation: one
            // byte permute packs two of them), lo = the value minus hi, rounded to bf16; hi + lo carries 16
            // mantissa bits without a bias (a truncated lo: twice the error), products are accumulated in fp32.
            const uint32_t ta = tmem_rows + ((uint32_t)(16 * pass) << 16) + kColKeys;
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
              uint32_t pk[16];  // hi of the lo half, hi of the hi half, lo, lo: four words each
#pragma unroll
              for (int tk = 0; tk < 2; ++tk) {
                const float4 x4 = lds128(row[pass][2 * tk] + 16 * i);
                const float4 y4 = lds128(row[pass][2 * tk + 1] + 16 * i);
                const float rl1 = rad[pass][2 * tk], rh1 = rad[pass][2 * tk + 1];
                const float2 rl = f2(rl1, rl1), rh = f2(rh1, rh1);
                const float2 x0 = __fmul2_rn(f2(x4.x, x4.y), rl), x1 = __fmul2_rn(f2(x4.z, x4.w), rl);
                const float2 y0 = __fmul2_rn(f2(y4.x, y4.y), rh), y1 = __fmul2_rn(f2(y4.z, y4.w), rh);
                float2 v[2][2];  // [half][pair]
                if constexpr (ROT) {
                  const float4 c = cs[tk][i][0], sn = cs[tk][i][1];
                  const float2 c0 = f2(c.x, c.y), c1 = f2(c.z, c.w);
                  const float2 s0 = f2(sn.x, sn.y), s1 = f2(sn.z, sn.w);
                  // x cos - y sin needs a negated operand and the packed fma has no negate modifier: the
                  // negative radius gives -y for the price of two packed multiplies
                  const float2 rn = f2(-rh1, -rh1);
                  const float2 m0 = __fmul2_rn(f2(y4.x, y4.y), rn), m1 = __fmul2_rn(f2(y4.z, y4.w), rn);
                  v[0][0] = __ffma2_rn(m0, s0, __fmul2_rn(x0, c0));
                  v[0][1] = __ffma2_rn(m1, s1, __fmul2_rn(x1, c1));
                  v[1][0] = __ffma2_rn(x0, s0, __fmul2_rn(y0, c0));
                  v[1][1] = __ffma2_rn(x1, s1, __fmul2_rn(y1, c1));
                } else {
                  v[0][0] = x0; v[0][1] = x1; v[1][0] = y0; v[1][1] = y1;
                }
#pragma unroll
                for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                  for (int e2 = 0; e2 < 2; ++e2) {
                    const uint32_t a0 = __float_as_uint(v[hf][e2].x), a1 = __float_as_uint(v[hf][e2].y);
                    const uint32_t h0 = a0 & 0xFFFF0000u, h1 = a1 & 0xFFFF0000u;
                    const float2 l = __ffma2_rn(f2(__uint_as_float(h0), __uint_as_float(h1)), f2(-1.f, -1.f), v[hf][e2]);
                    pk[4 * hf + 2 * tk + e2] = __byte_perm(a0, a1, 0x7632);
                    const __nv_bfloat162 lb = __floats2bfloat162_rn(l.x, l.y);
                    pk[8 + 4 * hf + 2 * tk + e2] = *reinterpret_cast<const uint32_t*>(&lb);
                  }
              }
              // this chunk's cos/sin registers are free: fetch the next pass's
              if (more) issue_cs_chunk(i);
              tmem_st_16x256b_x4(ta + 32 * i, pk);
              if (pass == 1 && i == NCH / 2 - 1) keys_ready(kBarKeys);
            }
          } else {  // nothing stored here: keep the pipeline moving
            if (more) {
#pragma unroll
              for (int i = 0; i < NCH; ++i) issue_cs_chunk(i);
            }
            if (pass == 1) keys_ready(kBarKeys);
          }
        }
        if (dead) break;

        // ---- softmax: thread = token row (lanes 0..15: tile w, 16..31: tile w + 4) ----
        const int xs = w + ((lane >> 4) << 2), tok = lane & 15, ts = first_tile(k) + xs;
        TileMeta ms;
        ms.phys = -2; ms.where = 0;
        if (xs < width) ms = meta_of(k, xs);
        // rows without a token (past the page's count, or position -1) take no part
        bool valid = tok < meta_tokens(ms);
        if (valid) valid = 16 * meta_sub(ms) + tok < (int)lds_u8(stage_at(slot, xs) + meta_hdr(ms) + 1);
        if (ROT && valid) {
          const int pos = (int)lds32(stage_at(slot, xs) + kst_pos + 4 * tok);
          if (pos >= p.max_pos && p.status) atomicOr(p.status, SPHKV_ST_BAD_POSITION);
          valid = pos >= 0;
        }
        keys_ready(kBarKeys2);
        if (k + 1 < rounds) extract(k + 1, slot_n);
        if (!__all_sync(0xffffffffu, mbar_wait(bar + 8 * kBarLogits, par_logits))) { dead = true; break; }
        par_logits ^= 1;
        tc_fence_after();
        float d[16], s[HEADS];
        if (PACK)
          tmem_ld_x8(tmem_rows + kColLogits, d);
        else
          tmem_ld_x16(tmem_rows + kColLogits, d);
        tmem_wait_ld();
        bool over = false;
#pragma unroll
        for (int h = 0; h < HEADS; ++h) {
          s[h] = valid ? d[h] + d[HEADS + h] : -INFINITY;
          over = over || s[h] > m_ref[h] + kSlack;
          m_true[h] = fmaxf(m_true[h], s[h]);
        }
        if (EXTRA && ms.phys != -2) {
          const int lb = lb0 + (ts >> tpp_shift);
          const int64_t hq0 = (int64_t)b * p.Hq + (int64_t)hkv * a.grp;
          if (p.logits_out != nullptr && valid)
#pragma unroll
            for (int h = 0; h < HEADS; ++h)
              if (h < a.grp)
                p.logits_out[((hq0 + h) * p.max_blocks + lb) * N + 16 * (ts & (TPP - 1)) + tok] = s[h] * kLn2;
        }
        if (EXTRA && p.page_ml != nullptr) {
          // per-tile (max, sum) in the natural-log domain, reduced over the tile's 16 lanes
          float* dst = p.page_ml + ((int64_t)b * p.Hq + (int64_t)hkv * a.grp) * ml_head + ((int64_t)lb0 * TPP + ts) * 2;
#pragma unroll
          for (int h = 0; h < HEADS; ++h) {
            float tm = s[h];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
            float ls = tm == -INFINITY ? 0.f : fast_exp2(s[h] - tm);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, o);
            if (tok == h && h < a.grp && ms.phys != -2) {
              dst[h * ml_head] = tm * kLn2;
              dst[h * ml_head + 1] = ls;
            }
          }
        }
        // Does any row of the team pass its reference maximum?  The weights are computed while the other
        // warps answer; hardly ever are they computed again.
        auto team_arrive = [&]() { if (lane == 0) mbar_arrive(bar + 8 * kBarVote); };
        auto team_wait = [&]() -> bool {
          const bool ok = __all_sync(0xffffffffu, mbar_wait(bar + 8 * kBarVote, par_vote));
          par_vote ^= 1;
          return ok;
        };
        const uint32_t vote_row = votes + (k & 1) * 16;
        over = __any_sync(0xffffffffu, over);
        if (lane == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(vote_row + 4 * w), "r"((uint32_t)over) : "memory");
        team_arrive();
        float pv[HEADS];
#pragma unroll
        for (int h = 0; h < HEADS; ++h) pv[h] = fast_exp2(s[h] - (m_ref[h] == -INFINITY ? 0.f : m_ref[h]));
        if (!team_wait()) { dead = true; break; }
        const float4 vt = lds_f4(vote_row);
        const bool raise = (__float_as_uint(vt.x) | __float_as_uint(vt.y) | __float_as_uint(vt.z) | __float_as_uint(vt.w)) != 0;
        // the previous macro tile's V product is done: its weights may be overwritten, the accumulator read
        if (k > 0) {
          if (!__all_sync(0xffffffffu, mbar_wait(bar + 8 * kBarOut, par_out))) { dead = true; break; }
          par_out ^= 1;
        }
        if (raise) {
#pragma unroll
          for (int h = 0; h < HEADS; ++h) {
            float mine = s[h];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mine = fmaxf(mine, __shfl_xor_sync(0xffffffffu, mine, o));
            if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(wmax + 32 * w + 4 * h), "f"(mine) : "memory");
          }
          team_arrive();
          if (!team_wait()) { dead = true; break; }
          float alpha[HEADS];
#pragma unroll
          for (int h = 0; h < HEADS; ++h) {
            float m_new = m_ref[h];
#pragma unroll
            for (int q = 0; q < 4; ++q) m_new = fmaxf(m_new, __uint_as_float(lds32(wmax + 32 * q + 4 * h)));
            alpha[h] = m_new == -INFINITY ? 1.f : fast_exp2(m_ref[h] - m_new);
            l_run[h] *= alpha[h];
            m_ref[h] = m_new;
            pv[h] = fast_exp2(s[h] - (m_new == -INFINITY ? 0.f : m_new));
          }
          if (k > 0) {
            tc_fence_after();
            float o[16];
            tmem_ld_x16(tmem_rows + kColOut, o);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 16; ++c) o[c] *= alpha[c & (HEADS - 1)];
            tmem_st_x16(tmem_rows + kColOut, o);
            tmem_wait_st();
          }
        }
        // ---- weights into the MN-major operand layout: token rows of 16 bytes (eight columns), 8-token
        //      groups at 128 bytes, the second eight columns at 256.  Hi + lo parts for either type of V: against
        //      a lagging reference maximum not even the largest weight is exactly 1, and 11 bits of it showed
        //      (error of a three-row step with f16 V against float64: 1.4e-4, so 1.3e-5; 24.6 -> 25.1 us) ----
#pragma unroll
        for (int h = 0; h < HEADS; ++h) l_run[h] += pv[h];
        if (xs < width) {
          uint32_t hi[HEADS / 2], lo[HEADS / 2];
#pragma unroll
          for (int h = 0; h < HEADS; h += 2) {
            if (kBf16)
              split_bf16x2(pv[h], pv[h + 1], hi[h / 2], lo[h / 2]);
            else
              split_f16x2(pv[h], pv[h + 1], hi[h / 2], lo[h / 2]);
          }
          const uint32_t dst = p_buf + xs * 512 + (tok >> 3) * 128 + (tok & 7) * 16;
          if (PACK) {
            sts128(dst, hi[0], hi[1], lo[0], lo[1]);
          } else {
            sts128(dst, hi[0], hi[1], hi[HEADS / 2 - 2], hi[HEADS / 2 - 1]);
            sts128(dst + 256, lo[0], lo[1], lo[HEADS / 2 - 2], lo[HEADS / 2 - 1]);
          }
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar + 8 * kBarWeights);
      }
      if (!dead) {
        if (!__all_sync(0xffffffffu, mbar_wait(bar + 8 * kBarOut, par_out))) dead = true;
        par_out ^= 1;
      }
      if (dead) tmem_wait_st();  // this warp's stores to tensor memory
    }
    if (dead) give_up();

    // ---- merge the teams of this CTA and write one partial row.  The accumulators [HEADS][DH] go where the
    //      weights were (the first eight columns of a packed tile: the zero columns stay) ----
    auto acc_at = [&](int t, int e) -> float* {
      return reinterpret_cast<float*>(smem + smem_head_bytes(DH) + t * smem_team_bytes(DH) + smem_v_bytes(DH) + (PACK ? (e >> 6) * 512 + (e & 63) * 4 : e * 4));
    };
    if (in_use) {
      const int w = warp & 3;
      float o[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) o[c] = 0.f;
      if (rounds > 0 && !dead) {
        tc_fence_after();
        tmem_ld_x16(tmem + ((uint32_t)(32 * w) << 16) + kColOut, o);
        tmem_wait_ld();
        tc_fence_before();
      }
#pragma unroll
      for (int h = 0; h < HEADS; ++h) {
        float l = l_run[h], m = m_true[h];
#pragma unroll
        for (int q = 16; q > 0; q >>= 1) {
          l += __shfl_xor_sync(0xffffffffu, l, q);
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, q));
        }
        if (lane == 0) {
          stats_of(team)[(w * 8 + h) * 2] = l;
          stats_of(team)[(w * 8 + h) * 2 + 1] = dead ? -INFINITY : m;
          if (w == 0) mref_of(team)[h] = dead ? -INFINITY : m_ref[h];
        }
        if (32 * w + lane < DH) *acc_at(team, h * DH + 32 * w + lane) = o[h] + o[h + HEADS];
      }
    }
    teams_barrier();
    dead = dead || shared_words[1] != 0;
    {
      float* out_row = a.rows + (int64_t)(blockIdx.x + u) * 8 * (DH + 2);
      for (int i = threadIdx.x; i < a.grp * DH; i += kTeamThreads) {
        const int n = i / DH, d = i % DH;
        float M = -INFINITY, L = 0.f, o = 0.f;
#pragma unroll
        for (int tw = 0; tw < 4 * kTeams; ++tw)
          if (tw < 4 * a.teams) M = fmaxf(M, stats_of(tw >> 2)[((tw & 3) * 8 + n) * 2 + 1]);
        if (M != -INFINITY) {
#pragma unroll
          for (int t = 0; t < kTeams; ++t) {
            if (t >= a.teams) break;
            const float mw = mref_of(t)[n];
            if (mw == -INFINITY) continue;
            const float sc = fast_exp2(mw - M);
            o += *acc_at(t, i) * sc;
            if (d == 0) {
              float l = 0.f;
#pragma unroll
              for (int w = 0; w < 4; ++w) l += stats_of(t)[(w * 8 + n) * 2];
              L += l * sc;
            }
          }
        }
        float* dst = out_row + n * (DH + 2);
        dst[2 + d] = o;
        if (d == 0) {
          dst[0] = M;
          dst[1] = L;
        }
      }
    }
  }
  }
  tc_fence_before();
  cta_barrier();
  if (warp == 4 * kTeams + 3) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace sphkv
