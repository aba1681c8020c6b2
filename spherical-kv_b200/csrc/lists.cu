// Page lists on the device: the grouping of retained tokens into pages that build_page_lists
// describes (the grouping and sort of _build_per_head_pages, spherical_kv_pipeline.py:1146-1228,
// and the pointer table of pointer_table.py:4-21).
//
//   sphkv_page_lists_count   tokens per (unit, tier slot, chunk) -> pages, bundles, byte offsets of
//                            every (tier slot, unit) run; the four totals that size the outputs
//                            come back to the host (the one synchronisation of the construction)
//   sphkv_page_lists_fill    every table in one launch (two with a page permutation)
//
// Bound: launches and the one round trip, not bandwidth (a 32768-token, 8-head prompt is 0.26 MB of
// tiers in and 2.5 MB of tables out).  As array operations the same construction was ~130 launches
// with 15 synchronising copies, 1.8 ms whatever the prompt's length.
#include <algorithm>

#include "common.cuh"

namespace sphkv {

constexpr int kListThreads = 256;
constexpr int kListPer = 8;                           // tokens per thread
constexpr int kListChunk = kListThreads * kListPer;   // tokens per CTA
constexpr int kScanThreads = 1024;
constexpr int kScanRuns = 1024;                       // runs whose token counts the scan keeps in shared memory
// The four totals go to the host as words that carry the number of the call in their upper 16 bits, so that each
// says by itself that it has arrived.  The byte total can need more than the other 48 (a large page_align): it stays at
// their largest value then, which is refused like any pool past 32-bit offsets.
constexpr int kTotalBits = 48;
constexpr int64_t kTotalMax = (INT64_C(1) << kTotalBits) - 1;

struct ListArgs {
  const void* assign;  // [U][T] tier ids
  int64_t T;
  int elem_size;       // bytes of a tier id: 1 (unsigned), 4 or 8
  int U, Hkv, S, n_chunks, N, n_shift, rb, align;
  int tier_id[SPHKV_MAX_TIER_SLOTS], G[SPHKV_MAX_TIER_SLOTS], bits[SPHKV_MAX_TIER_SLOTS];
  // scratch; run r = slot * U + unit
  int64_t* totals;     // pinned host memory: pages, most blocks of a unit, bundles, pool bytes (see kTotalBits)
  int64_t call;
  int64_t* byte_base;  // [S*U] pool offset of the run's first page
  int32_t* cnt;        // [S*U] tokens
  int32_t* run_base;   // [S*U] first logical page
  int32_t* bun_base;   // [S*U] first bundle
  int32_t* col_base;   // [S*U] first column in the unit's block list
  int32_t* chunk_cnt;  // [S*U][n_chunks] tokens per chunk, then their exclusive prefix
};

struct ListOut {
  int32_t *positions, *src_index, *page_head, *page_slot, *page_count, *ptable;
  int32_t *block_table, *bits_table, *num_blocks, *bundles;
  const int64_t* perm;  // physical page of every logical page; NULL = the same
  int max_blocks;
};

__device__ __forceinline__ int64_t page_bytes(const ListArgs& a, int s, int count) {
  // 32-bit arithmetic: a page is at most a few KB (a 64-bit division here was a third of the scan)
  const uint32_t vals = (uint32_t)count * a.G[s];
  const uint32_t b = 8 + 4 * a.G[s] + ((vals * a.bits[s] + 7) >> 3) + vals * a.rb;
  return (b + a.align - 1) / (uint32_t)a.align * a.align;
}

// tier ids of this thread's kListPer tokens (consecutive; INT64_MIN past the end: ids are
// compared as int64, and no slot's 32-bit id equals it)
__device__ __forceinline__ void load_tiers(const ListArgs& a, int u, int64_t t0, int64_t (&v)[kListPer]) {
  const int64_t base = (int64_t)u * a.T + t0;
  const char* p = reinterpret_cast<const char*>(a.assign) + base * a.elem_size;
  if (a.elem_size == 1 && t0 + kListPer <= a.T && (reinterpret_cast<uintptr_t>(p) & 7) == 0) {
    const uint2 w = __ldg(reinterpret_cast<const uint2*>(p));
#pragma unroll
    for (int e = 0; e < kListPer; ++e) v[e] = ((e < 4 ? w.x : w.y) >> (8 * (e & 3))) & 0xFFu;
    return;
  }
#pragma unroll
  for (int e = 0; e < kListPer; ++e) {
    if (t0 + e >= a.T)
      v[e] = INT64_MIN;
    else if (a.elem_size == 1)
      v[e] = reinterpret_cast<const uint8_t*>(p)[e];
    else if (a.elem_size == 4)
      v[e] = reinterpret_cast<const int32_t*>(p)[e];
    else
      v[e] = reinterpret_cast<const int64_t*>(p)[e];
  }
}
__device__ __forceinline__ uint32_t slot_mask(const ListArgs& a, int s, const int64_t (&v)[kListPer]) {
  uint32_t m = 0;
#pragma unroll
  for (int e = 0; e < kListPer; ++e) m |= (v[e] == (int64_t)a.tier_id[s] ? 1u : 0u) << e;
  return m;
}

// grid (chunk, unit)
__global__ void __launch_bounds__(kListThreads) list_count_kernel(const ListArgs a) {
  __shared__ int s_cnt[SPHKV_MAX_TIER_SLOTS];
  const int chunk = blockIdx.x, u = blockIdx.y, lane = threadIdx.x & 31;
  if (threadIdx.x < SPHKV_MAX_TIER_SLOTS) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  griddep_launch();
  int64_t v[kListPer];
  load_tiers(a, u, (int64_t)chunk * kListChunk + threadIdx.x * kListPer, v);
  for (int s = 0; s < a.S; ++s) {
    const int n = __reduce_add_sync(0xffffffffu, __popc(slot_mask(a, s, v)));
    if (lane == 0 && n) atomicAdd(&s_cnt[s], n);
  }
  __syncthreads();
  if ((int)threadIdx.x < a.S)
    a.chunk_cnt[((int64_t)threadIdx.x * a.U + u) * a.n_chunks + chunk] = s_cnt[threadIdx.x];
}

// Exclusive prefix over the CTA of one value per thread; `total` = the sum over all threads.
template <typename T>
__device__ __forceinline__ T block_exclusive(T v, T* s_part, T& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_part[warp] = x;
  __syncthreads();
  T before = 0;
  total = 0;
  for (int w = 0; w < nw; ++w) {
    const T p = s_part[w];
    if (w < warp) before += p;
    total += p;
  }
  __syncthreads();
  return before + x - v;
}

// one CTA: run r = slot * U + unit by thread
__global__ void __launch_bounds__(kScanThreads) list_scan_kernel(const ListArgs a) {
  __shared__ int64_t s_part[kScanThreads / 32];
  __shared__ int s_max[kScanThreads / 32];
  __shared__ int s_n[kScanRuns];
  griddep_wait();
  const int n_runs = a.S * a.U, ppb = 128 >> a.n_shift;
  int64_t c_pages = 0, c_bundles = 0, c_bytes = 0;
  for (int r0 = 0; r0 < n_runs; r0 += blockDim.x) {
    const int r = r0 + threadIdx.x;
    int n = 0;
    if (r < n_runs) {
      int32_t* cc = a.chunk_cnt + (int64_t)r * a.n_chunks;
      for (int c0 = 0; c0 < a.n_chunks; c0 += 8) {  // eight loads in flight
        int v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = c0 + e < a.n_chunks ? cc[c0 + e] : 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (c0 + e < a.n_chunks) cc[c0 + e] = n;
          n += v[e];
        }
      }
    }
    const int s = r < n_runs ? r / a.U : 0;
    const int pages = (n + a.N - 1) >> a.n_shift;
    const int64_t bytes =
        pages == 0 ? 0 : (pages - 1) * page_bytes(a, s, a.N) + page_bytes(a, s, n - ((pages - 1) << a.n_shift));
    // pages and bundles share one word: both stay below 2^31
    int64_t t_pb, t_bytes;
    const int64_t x_pb = block_exclusive<int64_t>(((int64_t)pages << 32) | (int64_t)((pages + ppb - 1) / ppb), s_part, t_pb);
    const int64_t x_bytes = block_exclusive<int64_t>(bytes, s_part, t_bytes);
    if (r < n_runs) {
      if (n_runs <= kScanRuns) s_n[r] = n;
      a.cnt[r] = n;
      a.run_base[r] = (int32_t)(c_pages + (x_pb >> 32));
      a.bun_base[r] = (int32_t)(c_bundles + (x_pb & 0xFFFFFFFFLL));
      a.byte_base[r] = c_bytes + x_bytes;
    }
    c_pages += t_pb >> 32;
    c_bundles += t_pb & 0xFFFFFFFFLL;
    c_bytes += t_bytes;
  }
  __syncthreads();
  const int* counts = n_runs <= kScanRuns ? s_n : a.cnt;
  int most = 0;
  for (int u = threadIdx.x; u < a.U; u += blockDim.x) {
    int col = 0;
    for (int s = 0; s < a.S; ++s) {
      a.col_base[s * a.U + u] = col;
      col += (counts[s * a.U + u] + a.N - 1) >> a.n_shift;
    }
    most = max(most, col);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = most;
  __syncthreads();
  if (threadIdx.x < 4) {  // the host polls these words
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) most = max(most, s_max[w]);
    const int64_t v = threadIdx.x == 0 ? c_pages : threadIdx.x == 1 ? most : threadIdx.x == 2 ? c_bundles : c_bytes + 16;
    *reinterpret_cast<volatile int64_t*>(a.totals + threadIdx.x) = min(v, kTotalMax) | (int64_t)((uint64_t)a.call << kTotalBits);
  }
}

// grid (chunk, unit): the chunk's tokens are compacted per tier slot in shared memory (order kept) and
// written out in rank order, so neighbouring threads write neighbouring page slots; the unit's page
// records are dealt out over its chunks' threads.
__global__ void __launch_bounds__(kListThreads) list_fill_kernel(const ListArgs a, const ListOut o) {
  __shared__ uint16_t s_tok[kListChunk];
  __shared__ int s_part[kListThreads / 32];
  __shared__ int s_run[SPHKV_MAX_TIER_SLOTS][5];  // tokens, first page, bundle and column, tokens before this chunk
  __shared__ int64_t s_byte[SPHKV_MAX_TIER_SLOTS];
  const int chunk = blockIdx.x, u = blockIdx.y, tid = threadIdx.x;
  const int N = a.N, ppb = 128 >> a.n_shift;
  griddep_launch();
  // what the loop over the slots reads of the scan: one latency instead of one per slot and use
  if (tid < 32 * SPHKV_MAX_TIER_SLOTS && (tid >> 5) < a.S) {
    const int s = tid >> 5, r = s * a.U + u, e = tid & 31;
    const int32_t* from = e == 0 ? a.cnt : e == 1 ? a.run_base : e == 2 ? a.bun_base : a.col_base;
    if (e < 4) s_run[s][e] = from[r];
    if (e == 4) s_run[s][4] = a.chunk_cnt[(int64_t)r * a.n_chunks + chunk];
    if (e == 5) s_byte[s] = a.byte_base[r];
  }
  const int64_t t_first = (int64_t)chunk * kListChunk;
  const int64_t row_first = (int64_t)(u / a.Hkv) * a.T;
  int64_t v[kListPer];
  load_tiers(a, u, t_first + tid * kListPer, v);
  __syncthreads();
  auto phys = [&](int64_t lp) -> int64_t { return o.perm != nullptr ? o.perm[lp] : lp; };
  int nb = 0;
  for (int s = 0; s < a.S; ++s) {
    const int n = s_run[s][0], pages = (n + N - 1) >> a.n_shift, base = s_run[s][1];
    uint32_t m = slot_mask(a, s, v);
    int mine;
    int at = block_exclusive<int>(__popc(m), s_part, mine);  // its barriers also order s_tok between slots
    while (m) {
      s_tok[at++] = (uint16_t)(tid * kListPer + __ffs(m) - 1);
      m &= m - 1;
    }
    __syncthreads();
    const int rank0 = s_run[s][4];
    for (int i = tid; i < mine; i += kListThreads) {
      const int rank = rank0 + i;
      const int64_t t = t_first + s_tok[i];
      const int64_t dst = (phys(base + (rank >> a.n_shift)) << a.n_shift) + (rank & (N - 1));
      o.positions[dst] = (int32_t)t;
      o.src_index[dst] = (int32_t)(row_first + t);
    }
    // empty slots of the run's last page
    if (chunk == 0 && n + tid < (pages << a.n_shift)) {
      const int64_t dst = (phys(base + pages - 1) << a.n_shift) + ((n + tid) & (N - 1));
      o.positions[dst] = -1;
      o.src_index[dst] = -1;
    }
    const int64_t full = page_bytes(a, s, N);
    for (int p = chunk * kListThreads + tid; p < pages; p += a.n_chunks * kListThreads) {
      const int64_t ph = phys(base + p);
      const int count = min(N, n - (p << a.n_shift));
      o.page_head[ph] = u % a.Hkv;
      o.page_slot[ph] = s;
      o.page_count[ph] = count;
      if (o.perm != nullptr) {
        o.ptable[3 * ph] = (int32_t)page_bytes(a, s, count);  // list_offsets_kernel turns sizes into offsets
      } else {
        const int64_t off = s_byte[s] + p * full, th = off + 8 + 4 * a.G[s];
        o.ptable[3 * ph] = (int32_t)off;
        o.ptable[3 * ph + 1] = (int32_t)th;
        o.ptable[3 * ph + 2] = (int32_t)(th + (((int64_t)count * a.G[s] * a.bits[s] + 7) >> 3));
      }
      const int64_t cell = (int64_t)u * o.max_blocks + s_run[s][3] + p;
      o.block_table[cell] = (int32_t)ph;
      o.bits_table[cell] = s;
      int32_t* bun = o.bundles + 8 * ((int64_t)s_run[s][2] + p / ppb);
      bun[p % ppb] = (int32_t)ph;
      if (p == pages - 1 || p % ppb == ppb - 1)  // the record's last page clears what follows it
        for (int e = p % ppb + 1; e < 8; ++e) bun[e] = -1;
    }
    nb += pages;
  }
  for (int c = nb + chunk * kListThreads + tid; c < o.max_blocks; c += a.n_chunks * kListThreads) {
    o.block_table[(int64_t)u * o.max_blocks + c] = -1;
    o.bits_table[(int64_t)u * o.max_blocks + c] = 0;
  }
  if (chunk == 0 && tid == 0) o.num_blocks[u] = nb;
}

// one CTA: pages in physical order, sizes -> offsets (only with a page permutation)
__global__ void __launch_bounds__(kScanThreads) list_offsets_kernel(const ListArgs a, const ListOut o, int n_pages) {
  __shared__ int64_t s_part[kScanThreads / 32];
  constexpr int kPer = 8;
  int64_t carry = 0;
  for (int64_t p0 = 0; p0 < n_pages; p0 += kScanThreads * kPer) {
    const int64_t first = p0 + threadIdx.x * kPer;
    int size[kPer];
    int64_t sum = 0;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      size[e] = first + e < n_pages ? o.ptable[3 * (first + e)] : 0;
      sum += size[e];
    }
    int64_t total;
    int64_t off = carry + block_exclusive<int64_t>(sum, s_part, total);
    carry += total;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      if (first + e < n_pages) {
        const int s = o.page_slot[first + e];
        const int64_t th = off + 8 + 4 * a.G[s];
        o.ptable[3 * (first + e)] = (int32_t)off;
        o.ptable[3 * (first + e) + 1] = (int32_t)th;
        o.ptable[3 * (first + e) + 2] = (int32_t)(th + (((int64_t)o.page_count[first + e] * a.G[s] * a.bits[s] + 7) >> 3));
      }
      off += size[e];
    }
  }
}

// The scan writes the four totals straight into pinned host memory: one small buffer per calling thread, freed
// with it.
struct PinnedTotals {
  int64_t* p = nullptr;
  int64_t calls = 0;
  int64_t* get() {
    if (p == nullptr) {
      if (cudaHostAlloc(reinterpret_cast<void**>(&p), 4 * sizeof(int64_t), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess)
        p = nullptr;
      else
        p[0] = p[1] = p[2] = p[3] = 0;
    }
    return p;
  }
  ~PinnedTotals() {
    if (p != nullptr) (void)cudaFreeHost(p);
  }
};

static int64_t list_chunks(int64_t T) { return (T + kListChunk - 1) / kListChunk; }

}  // namespace sphkv

using namespace sphkv;

extern "C" int64_t sphkv_page_lists_scratch_bytes(int32_t units, int64_t T, int32_t n_slots) {
  if (units <= 0 || T <= 0 || n_slots <= 0) return SPHKV_E_ARG;
  const int64_t runs = (int64_t)units * n_slots;
  return runs * (8 + 16) + runs * list_chunks(T) * 4;
}

static int list_args(ListArgs& a, const sphkv_page_lists_params* p) {
  SPHKV_REQUIRE(p != nullptr && p->tier_assign && p->scratch, SPHKV_E_ARG, "page_lists: NULL pointer");
  SPHKV_REQUIRE(p->units > 0 && p->Hkv > 0 && p->units % p->Hkv == 0 && p->T > 0 && p->units <= 65535, SPHKV_E_ARG,
                "page_lists: units=%d Hkv=%d T=%lld", p->units, p->Hkv, (long long)p->T);
  SPHKV_REQUIRE(p->page_size == 16 || p->page_size == 32 || p->page_size == 64 || p->page_size == 128, SPHKV_E_ARG,
                "page_lists: page_size=%d (16, 32, 64 or 128)", p->page_size);
  SPHKV_REQUIRE(p->elem_size == 1 || p->elem_size == 4 || p->elem_size == 8, SPHKV_E_DTYPE,
                "page_lists: tier ids of %d bytes (1, 4 or 8)", p->elem_size);
  SPHKV_REQUIRE(p->page_align >= 4 && p->page_align % 4 == 0, SPHKV_E_ARG, "page_lists: page_align=%d", p->page_align);
  SPHKV_REQUIRE(p->n_slots >= 1 && p->n_slots <= SPHKV_MAX_TIER_SLOTS, SPHKV_E_ARG, "page_lists: n_slots=%d", p->n_slots);
  SPHKV_REQUIRE((reinterpret_cast<uintptr_t>(p->scratch) & 15) == 0 &&
                    p->scratch_bytes >= sphkv_page_lists_scratch_bytes(p->units, p->T, p->n_slots),
                SPHKV_E_SCRATCH, "page_lists: scratch %lld B too small or misaligned", (long long)p->scratch_bytes);
  a.assign = p->tier_assign;
  a.T = p->T; a.elem_size = p->elem_size;
  a.U = p->units; a.Hkv = p->Hkv; a.S = p->n_slots;
  a.n_chunks = (int)list_chunks(p->T);
  a.N = p->page_size; a.n_shift = p->page_size == 16 ? 4 : p->page_size == 32 ? 5 : p->page_size == 64 ? 6 : 7;
  a.rb = p->radius_fmt == SPHKV_RADIUS_F16 ? 2 : 1;
  a.align = p->page_align;
  for (int s = 0; s < a.S; ++s) {
    SPHKV_REQUIRE(p->G[s] > 0 && p->bits[s] >= 1 && p->bits[s] <= 8, SPHKV_E_ARG, "page_lists: slot %d: G=%d bits=%d", s,
                  p->G[s], p->bits[s]);
    a.tier_id[s] = p->tier_id[s]; a.G[s] = p->G[s]; a.bits[s] = p->bits[s];
  }
  const int64_t runs = (int64_t)a.U * a.S;
  a.totals = nullptr;
  a.byte_base = reinterpret_cast<int64_t*>(p->scratch);
  a.cnt = reinterpret_cast<int32_t*>(a.byte_base + runs);
  a.run_base = a.cnt + runs;
  a.bun_base = a.run_base + runs;
  a.col_base = a.bun_base + runs;
  a.chunk_cnt = a.col_base + runs;
  return 0;
}

extern "C" int sphkv_page_lists_count(const sphkv_page_lists_params* p, int64_t* totals, void* stream) {
  ListArgs a;
  if (int rc = list_args(a, p)) return rc;
  SPHKV_REQUIRE(totals != nullptr, SPHKV_E_ARG, "page_lists_count: NULL pointer");
  static thread_local PinnedTotals pinned;
  int64_t* host = pinned.get();
  SPHKV_REQUIRE(host != nullptr, SPHKV_E_LIMIT, "page_lists_count: no pinned host memory");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  a.totals = host;
  a.call = ++pinned.calls;
  // as many warps as there are runs for (the prefix over the warps is serial)
  const int scan_threads = std::min(kScanThreads, (a.S * a.U + 31) / 32 * 32);
  list_count_kernel<<<dim3(a.n_chunks, a.U), kListThreads, 0, st>>>(a);
  (void)launch_overlapped(list_scan_kernel, dim3(1), dim3(scan_threads), 0, st, a);
  if (int rc = check_launch("page_lists_count")) return rc;
  // The host needs nothing but the totals, so it waits for these words, not for the stream.  An error, or a stream
  // that has ended without them, ends the wait.
  const auto arrived = [&]() {
    for (int i = 0; i < 4; ++i)
      if ((uint64_t)__atomic_load_n(host + i, __ATOMIC_ACQUIRE) >> kTotalBits != ((uint64_t)a.call & 0xFFFF)) return false;
    return true;
  };
  for (int64_t spins = 1; !arrived(); ++spins) {
    if (spins % 16384 != 0) continue;
    const cudaError_t e = cudaStreamQuery(st);
    if (e == cudaErrorNotReady || arrived()) continue;
    set_error("page_lists_count: %s", e == cudaSuccess ? "the totals did not arrive" : cudaGetErrorString(e));
    return e == cudaSuccess ? (int)cudaErrorUnknown : (int)e;
  }
  for (int i = 0; i < 4; ++i) totals[i] = host[i] & kTotalMax;
  return 0;
}

extern "C" int sphkv_page_lists_fill(const sphkv_page_lists_params* p, void* stream) {
  ListArgs a;
  if (int rc = list_args(a, p)) return rc;
  SPHKV_REQUIRE(p->positions && p->src_index && p->page_head && p->page_slot && p->page_count && p->ptable &&
                    p->block_table && p->bits_table && p->num_blocks && p->bundles && p->max_blocks > 0 && p->n_pages > 0,
                SPHKV_E_ARG, "page_lists_fill: NULL pointer or empty table");
  const ListOut o = {p->positions, p->src_index, p->page_head, p->page_slot, p->page_count, p->ptable,
                     p->block_table, p->bits_table, p->num_blocks, p->bundles, p->perm, p->max_blocks};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  list_fill_kernel<<<dim3(a.n_chunks, a.U), kListThreads, 0, st>>>(a, o);
  if (int rc = check_launch("list_fill_kernel")) return rc;
  if (o.perm != nullptr) {
    list_offsets_kernel<<<1, kScanThreads, 0, st>>>(a, o, p->n_pages);
    return check_launch("list_offsets_kernel");
  }
  return 0;
}
