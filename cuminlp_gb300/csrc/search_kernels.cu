// search_kernels.cu -- the device half of the batched branch-and-bound:
// parent selection, the branching policy, prune + compaction (c) and the
// box pool with eviction (d).  Every kernel reads the iteration's sizes
// from SolverDev, so one captured graph replays any iteration.
//
// The reference keeps its frontier on the host: a binary heap of 40-byte
// nodes and a refcounted box history (search/frontier.hpp:152-338,
// search/history.hpp:20-137), pruned by an O(N) host loop after every
// launch (search/driver.hpp:303-352).  Here the frontier is a pool of SoA
// boxes in HBM; selection is a radix select on the lower-bound keys, and
// every compaction is a stable, deterministic block scan.
#include <cfloat>
#include <cstdint>

#include "eval_core.cuh"
#include "launch.hpp"
#include "policy.cuh"
#include "search.hpp"
#include "stamps.cuh"

namespace cmn {

__device__ __forceinline__ bool gap_closed_dev(double gub, double bound, double tol)
{
  return __dsub_rn(gub, bound) <= __dmul_rn(tol, fmax(1.0, fabs(gub)));
}

__device__ __forceinline__ double key_to_lb(uint64_t k)
{
  const uint64_t u = (k >> 63) ? (k & 0x7fffffffffffffffULL) : ~k;
  return __longlong_as_double((long long)u);
}

// ---------------------------------------------------------------------
// init / begin / finish
// ---------------------------------------------------------------------
__global__ void init_kernel(const SolverCfg cfg, const SolverBufs b, const double* __restrict__ root_lb,
                            const double* __restrict__ root_ub, double gub0)
{
  const int t = threadIdx.x + blockIdx.x * blockDim.x;
  for (int v = t; v < cfg.n_vars; v += blockDim.x * gridDim.x) {  // the root box in store slot 0
    const double lo = root_lb[v], hi = root_ub[v];
    b.lo[v] = lo;
    b.hi[v] = hi;
    // and staged: the first iteration's parent
    const uint64_t at = (uint64_t)v * cfg.e_max;
    b.plo[at] = lo;
    b.phi[at] = hi;
    if (b.plo32 != nullptr) {
      b.plo32[at] = __double2float_rd(lo);
      b.phi32[at] = __double2float_ru(hi);
    }
  }
  if (t == 0) {
    SolverDev* d = b.dev;
    memset(d, 0, sizeof(SolverDev));
    d->gub = gub0;
    d->glb = -DBL_MAX;
    d->dropped_lb_min = INFINITY;
    d->dropped_min_key = ~0ULL;
    b.lb[0][0] = -DBL_MAX;
    b.slot[0][0] = 0;
    b.depth[0] = 0;
    b.sel[0][0] = kSelParent;
    b.pdepth[0] = 0;
    d->pre_valid = 1;
    d->pre_k = 1;
    d->free_top = cfg.pstride - 1;
    d->pool_size = 1;
    d->pool_min_key = lb_key(-DBL_MAX);
    d->pool_max_key = lb_key(-DBL_MAX);
    d->parity = 0;
    d->use_screen = 1;
    d->counters.peak_frontier = 1;
  }
}

// every store slot but the root's is free; pops take the low slots first
__global__ void free_init_kernel(const SolverCfg cfg, const SolverBufs b)
{
  const uint64_t n = cfg.pstride - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    b.free_slots[i] = (uint32_t)(cfg.pstride - 1 - i);
}

// Top of the loop of search/driver.hpp:221-233: convergence of the least
// pending lower bound, the expansion budget, and this iteration's size.
__global__ void begin_kernel(const SolverCfg cfg, const SolverBufs b)
{
  SolverDev* d = b.dev;
  if (!begin_search(*d)) return;
  const uint64_t L = d->pool_size;
  if (L == 0) {
    d->done = 1;
    return;
  }
  const double m = key_to_lb(d->pool_min_key);
  if (gap_closed_dev(d->gub, m, cfg.tolerance)) {
    d->converged = 1;
    d->done = 1;
    return;
  }
  d->glb = m;
  if (d->expansions >= cfg.iter_limit || (cfg.batch_iter_limit && d->iterations >= cfg.batch_iter_limit)) {
    d->done = 1;
    return;
  }
  uint64_t E = L < cfg.e_max ? L : cfg.e_max;
  const uint64_t left = cfg.iter_limit - d->expansions;
  if (E > left) E = left;
  const uint64_t t = now_ns();
  for (int i = 0; i < 8; ++i) d->stamps[i] = t;
  // the previous iteration's rebuild (the first one: init_kernel) staged the E
  // best entries of this pool
  if (!d->pre_valid || d->pre_k != E) d->error = 1;
  d->pre_valid = 0;
  d->pre_k = 0;
  d->pre_count = 0;
  d->iterations += 1;
  d->n_parents = E;
  d->n_children = E << cfg.log2C;
  d->salt_base = d->expansions;
  d->expansions += E;
  d->certify_count = 0;
  d->iter_valid = 0;
  d->iter_excluded = 0;
  d->remaining = 0;
  d->kept = 0;
  d->new_size = 0;
  d->child_min_key = ~0ULL;
  d->child_max_key = 0;
  d->extent = 0;
  d->survivors = 0;
  d->evict = 0;
  d->improved = 0;
  d->counters.iterations = d->iterations;
  d->counters.expansions = d->expansions;
}

// ---------------------------------------------------------------------
// radix select of the k-th smallest lower-bound key
// ---------------------------------------------------------------------
// over the current buffer after the children were appended behind the pool
// (n = extent), alive entries only: target 0 the cap (when evicting), target 1
// the next iteration's parents

// one of the two pool buffers without indexing the parameter arrays by a
// runtime value (which would copy them to local memory)
template <class T>
__device__ __forceinline__ T* parity_buf(T* const (&a)[2], uint32_t p)
{
  return p ? a[1] : a[0];
}

__device__ __forceinline__ const double* pool_lb(const SolverBufs& b) { return parity_buf(b.lb, b.dev->parity); }
__device__ __forceinline__ uint8_t* pool_sel(const SolverBufs& b) { return parity_buf(b.sel, b.dev->parity); }

__device__ __forceinline__ bool target_live(const RadixState& r)
{
  return r.active && !r.settled && r.bits_left != 0;
}

__device__ void radix_init(const SolverCfg& cfg, const SolverBufs& b)
{
  const SolverDev* d = b.dev;
  for (int t = 0; t < 2; ++t) {
    RadixState* rs = b.radix + t;
    const uint64_t k = t == 0 ? cfg.cap : d->pre_k;
    const bool active = (t == 0 ? d->evict != 0 : k > 0) && k < d->new_size;
    for (int i = threadIdx.x; i < kRadixBins; i += blockDim.x) rs->hist[i] = 0;
    if (threadIdx.x == 0) {
      const uint64_t lo = d->evict_lo_key, hi = d->evict_hi_key;
      const int common = lo <= hi ? ((lo ^ hi) == 0 ? 64 : __clzll((long long)(lo ^ hi))) : 0;
      const uint64_t top = common == 0 ? 0 : (~0ULL << (64 - common));
      rs->prefix = lo & top;
      rs->mask = top;
      rs->k = k;
      rs->less = 0;
      rs->active = active ? 1u : 0u;
      rs->settled = 0;
      rs->rank = active ? 1u : 0u;
      rs->bits_left = (uint32_t)(64 - common);
    }
  }
}

// Picks the digit whose bin holds the k-th entry: a scan over the bins by one
// block of kScanBlock threads. When the entries up to and including that bin are
// exactly k, the bin is taken whole and the search stops.
__device__ void radix_pick(const SolverBufs& b, RadixState* rs)
{
  constexpr int kPer = kRadixBins / kScanBlock;
  __shared__ uint64_t warp_sum[kScanBlock / 32];
  __shared__ int pick_d;
  __shared__ uint64_t pick_cum, pick_cnt;
  const int bits = rs->bits_left < (uint32_t)kRadixBits ? (int)rs->bits_left : kRadixBits;
  const int shift = (int)rs->bits_left - bits;
  const int nb = 1 << bits;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  uint32_t c[kPer];
  uint64_t x = 0;
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    c[e] = t * kPer + e < nb ? __ldcg(&rs->hist[t * kPer + e]) : 0u;
    x += c[e];
  }
  const uint64_t own = x;
  if (t == 0) pick_d = -1;
  for (int off = 1; off < 32; off <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) warp_sum[wid] = x;
  __syncthreads();
  uint64_t run = x - own;
  for (int w = 0; w < wid; ++w) run += warp_sum[w];
  const uint64_t k = rs->k;
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    if (run < k && k <= run + c[e]) {  // exactly one bin holds the k-th entry
      pick_d = t * kPer + e;
      pick_cum = run;
      pick_cnt = c[e];
    }
    run += c[e];
    if (t * kPer + e < nb) rs->hist[t * kPer + e] = 0;
  }
  __syncthreads();
  if (t == 0) {
    if (pick_d < 0) {  // fewer entries in the bucket than its rank: never expected
      b.dev->error = 1;
      rs->settled = 1;
      rs->rank = 0;
    } else {
      rs->less += pick_cum;
      rs->k = k - pick_cum;
      rs->prefix |= (uint64_t)pick_d << shift;
      rs->mask |= ((uint64_t)(nb - 1)) << shift;
      rs->bits_left = (uint32_t)shift;
      if (pick_cum + pick_cnt == k) {
        rs->settled = 1;
        rs->rank = 0;
      }
    }
  }
  __syncthreads();
}

// One digit's histogram per live target over the entries inside its
// bucket, in one read of the keys; false when no target is live. Each thread
// counts a run of equal bins in registers and adds it to the block's shared
// histogram only when the bin changes: converging lower bounds share most
// leading digits, so a pass makes few shared-memory atomics instead of one per
// entry on one address.
__device__ __forceinline__ bool radix_hist(const SolverBufs& b, unsigned blocks, uint64_t n, uint32_t parity,
                                           bool (&go)[2])
{
  __shared__ uint32_t h[2][kRadixBins];
  int shift[2] = {0, 0}, nb[2] = {1, 1};
  uint64_t prefix[2] = {0, 0}, mask[2] = {0, 0};
  for (int t = 0; t < 2; ++t) {
    const RadixState& r = b.radix[t];
    go[t] = target_live(r);
    if (!go[t]) continue;
    const int bits = r.bits_left < (uint32_t)kRadixBits ? (int)r.bits_left : kRadixBits;
    shift[t] = (int)r.bits_left - bits;
    nb[t] = 1 << bits;
    prefix[t] = r.prefix;
    mask[t] = r.mask;
  }
  if (!go[0] && !go[1]) return false;
  // while both targets sit in the same bucket (the first pass of a rebuild)
  // their histograms are the same: count once, add to both
  const bool same = go[0] && go[1] && prefix[0] == prefix[1] && mask[0] == mask[1] && shift[0] == shift[1];
  const bool count1 = go[1] && !same;
  for (int t = 0; t < 2; ++t)
    for (int i = threadIdx.x; i < kRadixBins; i += blockDim.x) h[t][i] = 0;
  __syncthreads();
  const uint64_t* __restrict__ lb = reinterpret_cast<const uint64_t*>(parity_buf(b.lb, parity));
  const uint8_t* sel = parity_buf(b.sel, parity);
  const int lane = threadIdx.x & 31;
  // each warp takes chunks of 32 x kHistUnroll consecutive entries and
  // issues all their loads before it bins them
  constexpr int kChunk = 32 * kHistUnroll;
  const uint64_t warps = (uint64_t)blocks * (blockDim.x / 32);
  uint32_t run_bin[2] = {0, 0}, run[2] = {0, 0};
  for (uint64_t c = (uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); c * kChunk < n; c += warps) {
    uint64_t x[kHistUnroll];
    bool in[kHistUnroll];
#pragma unroll
    for (int u = 0; u < kHistUnroll; ++u) {
      const uint64_t i = c * kChunk + (uint64_t)u * 32 + lane;
      in[u] = i < n;
      x[u] = in[u] ? lb[i] : 0;
      if (in[u]) in[u] = sel[i] == kSelAlive;
    }
#pragma unroll
    for (int u = 0; u < kHistUnroll; ++u) {
      if (!in[u]) continue;
      const uint64_t key = bits_key(x[u]);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (!(t == 0 ? go[0] : count1) || (key & mask[t]) != prefix[t]) continue;
        const uint32_t bin = (uint32_t)(key >> shift[t]) & (uint32_t)(nb[t] - 1);
        if (bin != run_bin[t]) {
          if (run[t]) atomicAdd(&h[t][run_bin[t]], run[t]);
          run_bin[t] = bin;
          run[t] = 0;
        }
        ++run[t];
      }
    }
  }
  for (int t = 0; t < 2; ++t)
    if (run[t]) atomicAdd(&h[t][run_bin[t]], run[t]);
  __syncthreads();
  for (int t = 0; t < 2; ++t) {
    if (!go[t]) continue;
    const uint32_t* src = (t == 1 && same) ? h[0] : h[t];
    for (int i = threadIdx.x; i < nb[t]; i += blockDim.x)
      if (src[i]) atomicAdd(&b.radix[t].hist[i], src[i]);
  }
  return true;
}

// ---------------------------------------------------------------------
// stable compaction: count -> scan -> scatter over tiles of kScanTile
// items; item j of thread t in tile T is T * kScanTile + j * kScanBlock + t,
// so every pass reads whole cache lines and keeps kScanItems loads in flight
// per thread.
// ---------------------------------------------------------------------
// first item of this thread in a tile (by default its block's), read once per
// kernel (the special registers are slow to re-read)
__device__ __forceinline__ uint64_t tile_first(uint64_t tile) { return tile * kScanTile + threadIdx.x; }
__device__ __forceinline__ uint64_t tile_first() { return tile_first(blockIdx.x); }

__device__ __forceinline__ uint64_t tile_item(uint64_t t0, int j) { return t0 + (uint64_t)j * kScanBlock; }

// Ranks of the flagged items of this block's tile in item order (for every
// item: the flagged items before it); returns the tile's flagged count. One
// call per kernel and table slot `S`.
template <int S = 0>
__device__ __forceinline__ int tile_ranks(const bool (&f)[kScanItems], int (&rank)[kScanItems])
{
  constexpr int kWarps = kScanBlock / 32;
  constexpr int kPer = kScanItems * kWarps / 32;  // table entries per lane of warp 0
  __shared__ int tab[kScanItems * kWarps];
  __shared__ int tile_total;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned ball[kScanItems];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    ball[j] = __ballot_sync(0xffffffffu, f[j]);
    if (lane == 0) tab[j * kWarps + wid] = __popc(ball[j]);
  }
  __syncthreads();
  if (wid == 0) {
    int v[kPer], sum = 0;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      v[e] = tab[lane * kPer + e];
      sum += v[e];
    }
    int x = sum;
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    int run = x - sum;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      tab[lane * kPer + e] = run;
      run += v[e];
    }
    if (lane == 31) tile_total = x;
  }
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) rank[j] = tab[j * kWarps + wid] + __popc(ball[j] & lt);
  return tile_total;
}

// tile_ranks of two flag sets with one pair of barriers; their counts in `total`
__device__ __forceinline__ void tile_ranks2(const bool (&f)[kScanItems], const bool (&g)[kScanItems],
                                            int (&rf)[kScanItems], int (&rg)[kScanItems], int (&total)[2])
{
  constexpr int kWarps = kScanBlock / 32;
  constexpr int kPer = kScanItems * kWarps / 32;
  __shared__ int tab[2][kScanItems * kWarps];
  __shared__ int tile_total[2];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned bf[kScanItems], bg[kScanItems];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    bf[j] = __ballot_sync(0xffffffffu, f[j]);
    bg[j] = __ballot_sync(0xffffffffu, g[j]);
    if (lane == 0) {
      tab[0][j * kWarps + wid] = __popc(bf[j]);
      tab[1][j * kWarps + wid] = __popc(bg[j]);
    }
  }
  __syncthreads();
  if (wid < 2) {  // warp 0 scans the first table, warp 1 the second
    int* t = tab[wid];
    int v[kPer], sum = 0;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      v[e] = t[lane * kPer + e];
      sum += v[e];
    }
    int x = sum;
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    int run = x - sum;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      t[lane * kPer + e] = run;
      run += v[e];
    }
    if (lane == 31) tile_total[wid] = x;
  }
  __syncthreads();
  total[0] = tile_total[0];
  total[1] = tile_total[1];
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    rf[j] = tab[0][j * kWarps + wid] + __popc(bf[j] & lt);
    rg[j] = tab[1][j * kWarps + wid] + __popc(bg[j] & lt);
  }
}

__device__ __forceinline__ uint64_t warp_min_u64(uint64_t m)
{
  for (int off = 16; off > 0; off >>= 1) {
    const uint64_t o = __shfl_xor_sync(0xffffffffu, m, off);
    m = o < m ? o : m;
  }
  return m;
}

__device__ __forceinline__ uint64_t warp_max_u64(uint64_t m)
{
  for (int off = 16; off > 0; off >>= 1) {
    const uint64_t o = __shfl_xor_sync(0xffffffffu, m, off);
    m = o > m ? o : m;
  }
  return m;
}

// Sum of `c` over the block (one call per kernel and slot `S`).
template <int S = 0>
__device__ __forceinline__ int tile_count(int c)
{
  __shared__ int tot;
  if (threadIdx.x == 0) tot = 0;
  __syncthreads();
  const int w = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && w) atomicAdd(&tot, w);
  __syncthreads();
  return tot;
}

// Block totals of per-thread counters, for thread 0 (one global atomic per
// block instead of one per warp: same-address atomics serialise in L2).
// Every thread of the block calls it.
template <int N>
__device__ __forceinline__ void block_sum(unsigned long long (&v)[N])
{
  __shared__ unsigned long long acc[N];
  if (threadIdx.x < N) acc[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    unsigned long long x = v[k];
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd(&acc[k], x);
  }
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = acc[k];
}

// Block maximum of `m`, for thread 0. Every thread of the block calls it.
__device__ __forceinline__ uint64_t block_max(uint64_t m)
{
  __shared__ unsigned long long acc;
  if (threadIdx.x == 0) acc = 0;
  __syncthreads();
  for (int off = 16; off > 0; off >>= 1) {
    const uint64_t o = __shfl_down_sync(0xffffffffu, m, off);
    m = o > m ? o : m;
  }
  if ((threadIdx.x & 31) == 0 && m != 0) atomicMax(&acc, (unsigned long long)m);
  __syncthreads();
  return acc;
}

// Block minimum of `m`, for thread 0. Every thread of the block calls it.
__device__ __forceinline__ uint64_t block_min(uint64_t m)
{
  __shared__ unsigned long long acc;
  if (threadIdx.x == 0) acc = ~0ULL;
  __syncthreads();
  for (int off = 16; off > 0; off >>= 1) {
    const uint64_t o = __shfl_down_sync(0xffffffffu, m, off);
    m = o < m ? o : m;
  }
  if ((threadIdx.x & 31) == 0 && m != ~0ULL) atomicMin(&acc, (unsigned long long)m);
  __syncthreads();
  return acc;
}

// Exclusive scan of the tile counts of `*n_items` items (one block of 1024
// threads); writes the total to *total_out.
__global__ void __launch_bounds__(1024) scan_kernel(const uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets,
                                                    const uint64_t* __restrict__ n_items, uint64_t* total_out,
                                                    const uint32_t* __restrict__ done)
{
  __shared__ uint64_t warp_sum[32];
  if (*done) return;
  const uint64_t n = *n_items;
  const uint64_t nblocks = (n + kScanTile - 1) / kScanTile;
  // each thread sums a run of consecutive counts, the block scans the sums
  // once, and each thread writes its run's offsets: one pass, two barriers
  const uint32_t* src = counts;
  const uint64_t per = (nblocks + blockDim.x - 1) / blockDim.x;
  const uint64_t b0 = (uint64_t)threadIdx.x * per;
  const uint64_t b1 = b0 + per < nblocks ? b0 + per : nblocks;
  uint64_t sum = 0;
  for (uint64_t i = b0; i < b1; ++i) sum += src[i];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t x = sum;
  for (int off = 1; off < 32; off <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) warp_sum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint64_t w = lane < (int)(blockDim.x / 32) ? warp_sum[lane] : 0;
    for (int off = 1; off < 32; off <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += y;
    }
    warp_sum[lane] = w;  // inclusive
  }
  __syncthreads();
  uint64_t run = x - sum + (wid > 0 ? warp_sum[wid - 1] : 0);
  if (threadIdx.x == blockDim.x - 1) *total_out = run + sum;
  for (uint64_t i = b0; i < b1; ++i) {
    offsets[i] = (uint32_t)run;
    run += src[i];
  }
}

// ---- predicates / operations -----------------------------------------
struct KeptChild {
  SolverBufs b;
  __device__ bool operator()(uint64_t g) const
  {
    return b.cstate[g] == kChildEligible && !bits_lt(dbits(b.dev->gub), dbits(b.clb[g]));
  }
};

struct ScreenedChild {
  SolverBufs b;
  __device__ uint64_t size() const { return b.dev->n_children; }
  __device__ bool operator()(uint64_t g) const { return b.cstate[g] == kChildScreened; }
  __device__ bool skip() const { return b.dev->done != 0; }
};

template <class P>
__global__ void __launch_bounds__(kScanBlock) count_kernel(const P pred, uint32_t* __restrict__ counts)
{
  const uint64_t t0 = tile_first();
  if (pred.skip()) return;
  const uint64_t n = pred.size();
  if ((uint64_t)blockIdx.x * kScanTile >= n) return;
  bool f[kScanItems];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = tile_item(t0, j);
    f[j] = i < n && pred(i);
  }
  int c = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) c += f[j] ? 1 : 0;
  c = tile_count(c);
  if (threadIdx.x == 0) counts[blockIdx.x] = (uint32_t)c;
}

// The select decision of one target for one entry (`key` already masked).
struct TargetView {
  bool active, settled, ranked;
  uint64_t prefix, mask, k;
  __device__ explicit TargetView(const RadixState& r)
      : active(r.active != 0), settled(r.settled != 0), ranked(r.rank != 0), prefix(r.prefix), mask(r.mask), k(r.k)
  {
  }
  __device__ bool take(uint64_t key, bool eq, uint64_t eq_rank) const
  {
    if (!active) return true;
    if (eq) return settled || eq_rank < k;
    return (key & mask) < prefix;
  }
};

// stage the box in store slot `s` as parent `pos` of the staging planes
__device__ __forceinline__ void stage_parent(const SolverCfg& cfg, const SolverBufs& b, uint64_t s, uint64_t pos)
{
  if (pos >= cfg.e_max) {  // more marks than parents: never written, flagged
    b.dev->error = 1;
    return;
  }
  // loads in groups ahead of the stores (the pointers do not alias)
  const double* __restrict__ slo = b.lo + s * (uint64_t)cfg.n_vars;
  const double* __restrict__ shi = b.hi + s * (uint64_t)cfg.n_vars;
  double* __restrict__ plo = b.plo;
  double* __restrict__ phi = b.phi;
  const uint32_t dep = b.depth[s];
  constexpr int kGroup = 8;
  for (int v0 = 0; v0 < cfg.n_vars; v0 += kGroup) {
    double l[kGroup], h[kGroup];
#pragma unroll
    for (int u = 0; u < kGroup; ++u)
      if (v0 + u < cfg.n_vars) {
        l[u] = slo[v0 + u];
        h[u] = shi[v0 + u];
      }
#pragma unroll
    for (int u = 0; u < kGroup; ++u)
      if (v0 + u < cfg.n_vars) {
        const uint64_t at = (uint64_t)(v0 + u) * cfg.e_max + pos;
        plo[at] = l[u];
        phi[at] = h[u];
        if (b.plo32 != nullptr) {
          b.plo32[at] = __double2float_rd(l[u]);
          b.phi32[at] = __double2float_ru(h[u]);
        }
      }
  }
  b.pdepth[pos] = dep;
}

// decode a kept child from its parent into a free store slot and append it
// behind the pool in the current buffer (position pool_size + pos)
struct AppendChild {
  SolverCfg cfg;
  SolverBufs b;
  __device__ void operator()(uint64_t g, uint64_t pos) const
  {
    const SolverDev* d = b.dev;
    if (pos >= d->free_top) {  // more children than free slots: never expected
      b.dev->error = 1;
      return;
    }
    const uint64_t s = b.free_slots[d->free_top - 1 - pos];
    const uint64_t at = d->pool_size + pos;
    const uint32_t p = d->parity;
    const uint64_t k = g >> cfg.log2C, r = g & ((1ULL << cfg.log2C) - 1ULL);
    // every load is issued before the stores it does not depend on: the
    // pointers do not alias, and without that each parent value would wait
    // for the store before it
    const double* __restrict__ plo = b.plo;
    const double* __restrict__ phi = b.phi;
    double* __restrict__ slo = b.lo + s * (uint64_t)cfg.n_vars;
    double* __restrict__ shi = b.hi + s * (uint64_t)cfg.n_vars;
    const ParentInfo pi = b.pinfo[k];
    const double clb = b.clb[g];
    const uint32_t dep = b.pdepth[k];
    constexpr int kGroup = 8;
    for (int v0 = 0; v0 < cfg.n_vars; v0 += kGroup) {
      double l[kGroup], h[kGroup];
#pragma unroll
      for (int u = 0; u < kGroup; ++u)
        if (v0 + u < cfg.n_vars) {
          l[u] = plo[(uint64_t)(v0 + u) * cfg.e_max + k];
          h[u] = phi[(uint64_t)(v0 + u) * cfg.e_max + k];
        }
#pragma unroll
      for (int u = 0; u < kGroup; ++u)
        if (v0 + u < cfg.n_vars) {
          slo[v0 + u] = l[u];
          shi[v0 + u] = h[u];
        }
    }
    const SlotPlan* sp = b.slots + k * (uint64_t)cfg.max_slots;
    for (uint32_t j = 0; j < pi.count; ++j) {
      const SlotPlan sj = sp[j];
      const uint64_t part = slot_part(r, sj);
      double lo, hi;
      slot_bounds(sj, plo[(uint64_t)sj.vid * cfg.e_max + k], phi[(uint64_t)sj.vid * cfg.e_max + k], part, lo, hi);
      slo[sj.vid] = lo;
      shi[sj.vid] = hi;
    }
    b.depth[s] = dep + 1;
    parity_buf(b.lb, p)[at] = clb;
    parity_buf(b.slot, p)[at] = (uint32_t)s;
    parity_buf(b.sel, p)[at] = kSelAlive;
  }
};

struct ListChild {
  SolverBufs b;
  __device__ void operator()(uint64_t g, uint64_t pos) const { b.list[pos] = (uint32_t)g; }
};

template <class P, class Op>
__global__ void __launch_bounds__(kScanBlock) scatter_kernel(const P pred, const Op op,
                                                             const uint32_t* __restrict__ offsets)
{
  const uint64_t t0 = tile_first();
  if (pred.skip()) return;
  const uint64_t n = pred.size();
  if ((uint64_t)blockIdx.x * kScanTile >= n) return;
  bool f[kScanItems];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = tile_item(t0, j);
    f[j] = i < n && pred(i);
  }
  int rank[kScanItems];
  tile_ranks(f, rank);
  const uint64_t base = offsets[blockIdx.x];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j)
    if (f[j]) op(tile_item(t0, j), base + (uint64_t)rank[j]);
}

// appends the kept children listed (in order) by the compaction, one thread
// per child so that each child's chain of dependent loads runs in parallel
__global__ void append_children_kernel(const SolverCfg cfg, const SolverBufs b)
{
  const SolverDev* d = b.dev;
  if (halted(*d)) return;
  const uint64_t n = d->kept;
  const AppendChild op{cfg, b};
  for (uint64_t pos = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; pos < n; pos += (uint64_t)gridDim.x * blockDim.x)
    op(b.list[pos], pos);
}

// The same with G lanes per child, lane = variable: a box of the store is
// contiguous, so a child's bounds go out in whole lines, where one thread per
// child wrote 8 bytes of 32 lines at a time.  A group takes kAppendRun
// children in a row and keeps the parent's bounds in registers while they
// share it (the list is in parent order).  n = 64, 2^20 kept children (1.05 GB
// of boxes): 1.18 ms with one thread per child.  From nine variables on; below
// that a lane group would be mostly idle.
constexpr int kAppendRun = 16;
constexpr int kAppendVars = 2;  // variables a lane holds at a time

template <int G>
__global__ void __launch_bounds__(256) append_boxes_kernel(const SolverCfg cfg, const SolverBufs b)
{
  const SolverDev* d = b.dev;
  if (halted(*d)) return;
  const uint64_t kept = d->kept, free_top = d->free_top;
  const int n = cfg.n_vars;
  const int gl = threadIdx.x & (G - 1);
  const unsigned gmask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << ((threadIdx.x & 31) & ~(G - 1));
  const uint64_t groups = (uint64_t)gridDim.x * (blockDim.x / G);
  const uint32_t par = d->parity;
  const uint64_t pool = d->pool_size;
  if (kept > free_top) {  // more children than free slots: never expected
    if (threadIdx.x == 0 && blockIdx.x == 0) b.dev->error = 1;
    return;
  }
  for (uint64_t run = (uint64_t)blockIdx.x * (blockDim.x / G) + threadIdx.x / G; run * kAppendRun < kept; run += groups) {
    const uint64_t p0 = run * kAppendRun;
    const int cnt = kept - p0 < kAppendRun ? (int)(kept - p0) : kAppendRun;
    // lane = child: its store slot and the pool's entry
    uint32_t g_of[kAppendRun / G > 0 ? kAppendRun / G : 1], s_of[kAppendRun / G > 0 ? kAppendRun / G : 1];
#pragma unroll
    for (int u = 0; u < (kAppendRun / G > 0 ? kAppendRun / G : 1); ++u) {
      const int c = u * G + gl;
      g_of[u] = s_of[u] = 0;
      if (c < cnt) {
        const uint64_t pos = p0 + c;
        const uint32_t g = b.list[pos], s = b.free_slots[free_top - 1 - pos];
        g_of[u] = g;
        s_of[u] = s;
        b.depth[s] = b.pdepth[g >> cfg.log2C] + 1;
        parity_buf(b.lb, par)[pool + pos] = b.clb[g];
        parity_buf(b.slot, par)[pool + pos] = s;
        parity_buf(b.sel, par)[pool + pos] = kSelAlive;
      }
    }
    // lane = variable: the boxes
    for (int v0 = 0; v0 < n; v0 += G * kAppendVars) {
      uint32_t cur = 0xffffffffu;
      double lo[kAppendVars], hi[kAppendVars];
      const SlotPlan* plan[kAppendVars];  // the slot that narrows the variable, if any
      for (int c = 0; c < cnt; ++c) {
        uint32_t g = g_of[0], s = s_of[0];
#pragma unroll
        for (int u = 1; u < (kAppendRun / G > 0 ? kAppendRun / G : 1); ++u)
          if (c / G == u) g = g_of[u], s = s_of[u];
        g = __shfl_sync(gmask, g, c & (G - 1), G);
        s = __shfl_sync(gmask, s, c & (G - 1), G);
        const uint32_t k = g >> cfg.log2C;
        const uint64_t r = g & ((1u << cfg.log2C) - 1u);
        if (k != cur) {
          cur = k;
          const uint32_t count = b.pinfo[k].count;
          const SlotPlan* sp = b.slots + (uint64_t)k * cfg.max_slots;
#pragma unroll
          for (int u = 0; u < kAppendVars; ++u) {
            const int v = v0 + u * G + gl;
            plan[u] = nullptr;
            if (v < n) {
              lo[u] = b.plo[(uint64_t)v * cfg.e_max + k];
              hi[u] = b.phi[(uint64_t)v * cfg.e_max + k];
              for (uint32_t j = 0; j < count; ++j)
                if (sp[j].vid == (uint32_t)v) plan[u] = sp + j;  // the last one, as the slots are applied in order
            }
          }
        }
#pragma unroll
        for (int u = 0; u < kAppendVars; ++u) {
          const int v = v0 + u * G + gl;
          if (v >= n) continue;
          double l = lo[u], h = hi[u];
          if (plan[u] != nullptr) slot_bounds(*plan[u], lo[u], hi[u], slot_part(r, *plan[u]), l, h);
          b.lo[(uint64_t)s * n + v] = l;
          b.hi[(uint64_t)s * n + v] = h;
        }
      }
    }
  }
}

// pool entries [start, start + count) in position order, unpacked from the
// store
__global__ void frontier_gather_kernel(const SolverCfg cfg, const SolverBufs b, uint64_t start, uint64_t count,
                                       double* __restrict__ boxes, uint32_t* __restrict__ depths)
{
  const uint32_t p = b.dev->parity;
  const uint32_t* slot = parity_buf(b.slot, p);
  const int n = cfg.n_vars;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t s = slot[start + i];
    if (boxes)
      for (int v = 0; v < n; ++v) {
        boxes[(i * n + v) * 2] = b.lo[s * (uint64_t)cfg.n_vars + v];
        boxes[(i * n + v) * 2 + 1] = b.hi[s * (uint64_t)cfg.n_vars + v];
      }
    if (depths) depths[i] = b.depth[s];
  }
}

// ---------------------------------------------------------------------
// branching: BisectionBudgetCompositionPolicy::choose per parent
// ---------------------------------------------------------------------
// kLocal > 0: the policy's per-parent scratch lives in this thread's local
// memory (n <= kLocal), which the hardware interleaves across the warp and
// caches in L1; otherwise in the global scratch arrays
template <int kLocal>
__global__ void branch_kernel(const SolverCfg cfg, const SolverBufs b)
{
  const SolverDev* d = b.dev;
  if (d->done) return;
  const uint64_t E = d->n_parents;
  const int n = cfg.n_vars;
  const PolicyParams pp = {cfg.log2C, cfg.max_cycle, cfg.enumerate_cap, cfg.relative};
  const bool lazy = cfg.precision == CMN_PRECISION_FP32_LAZY;
  uint64_t fathomed = 0, fathomed_points = 0, bounded = 0;
  EnumCand ec_local[kLocal > 0 ? kLocal : 1];
  BisCand bc_local[kLocal > 0 ? kLocal : 1];
  uint64_t heap_local[kLocal > 0 ? kLocal : 1];
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < E; k += (uint64_t)gridDim.x * blockDim.x) {
    EnumCand* ec = kLocal > 0 ? ec_local : reinterpret_cast<EnumCand*>(b.enum_scratch) + k * (uint64_t)n;
    BisCand* bc = kLocal > 0 ? bc_local : reinterpret_cast<BisCand*>(b.bis_scratch) + k * (uint64_t)n;
    uint64_t* heap = kLocal > 0 ? heap_local : b.heap_scratch + k * (uint64_t)n;
    SlotPlan* sp = b.slots + k * (uint64_t)cfg.max_slots;
    ParentInfo pi = bisection_policy(b.plo + k, b.phi + k, cfg.e_max, n, b.kinds, pp, ec, bc, heap, sp);
    b.pinfo[k] = pi;
    // lazy form: the box's FP64 verdict runs beside this kernel, and
    // lazy_drop_kernel applies it and counts afterwards
    if (lazy) continue;
    if (pi.fathom) {
      ++fathomed;
      fathomed_points += pi.nreg;
    } else {
      bounded += pi.nreg;
    }
  }
  if (threadIdx.x == 0) stamp_last(b.dev->stamps + 1, (uint64_t)blockIdx.x * blockDim.x < E);
  if (lazy) return;  // every thread of the block takes this branch
  unsigned long long c[3] = {fathomed, fathomed_points, bounded};
  block_sum(c);
  if (threadIdx.x == 0) {
    if (c[0]) atomicAdd((unsigned long long*)&b.dev->counters.fathomed, c[0]);
    if (c[1]) atomicAdd((unsigned long long*)&b.dev->counters.fathomed_points, c[1]);
    if (c[2]) atomicAdd((unsigned long long*)&b.dev->counters.bounded, c[2]);
  }
}

// Lazy form, after the FP64 verdict of the staged parents (run beside the
// branching): a box that the reference predicate or the incumbent excludes
// is not expanded -- its plan becomes empty -- and the expansion counters
// are taken as branch_kernel takes them for the other forms.
__global__ void lazy_drop_kernel(const SolverCfg cfg, const SolverBufs b)
{
  const SolverDev* d = b.dev;
  if (d->done) return;
  const uint64_t E = d->n_parents;
  const double gub = d->gub;
  uint64_t fathomed = 0, fathomed_points = 0, bounded = 0, certified = 0, dropped = 0;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < E; k += (uint64_t)gridDim.x * blockDim.x) {
    ParentInfo pi = b.pinfo[k];
    ++certified;
    if (!b.pfeas[k] || b.plb[k] > gub) {
      pi = ParentInfo{0, 0, 0};
      b.pinfo[k] = pi;
      ++dropped;
    }
    if (pi.fathom) {
      ++fathomed;
      fathomed_points += pi.nreg;
    } else {
      bounded += pi.nreg;
    }
  }
  unsigned long long c[5] = {fathomed, fathomed_points, bounded, certified, dropped};
  block_sum(c);
  if (threadIdx.x == 0) {
    if (c[0]) atomicAdd((unsigned long long*)&b.dev->counters.fathomed, c[0]);
    if (c[1]) atomicAdd((unsigned long long*)&b.dev->counters.fathomed_points, c[1]);
    if (c[2]) atomicAdd((unsigned long long*)&b.dev->counters.bounded, c[2]);
    if (c[3]) atomicAdd((unsigned long long*)&b.dev->counters.certified_fp64, c[3]);
    if (c[4]) atomicAdd((unsigned long long*)&b.dev->counters.certify_pruned, c[4]);
  }
}

// Lazy form, per child, after lazy_drop_kernel: the FP32 pass wrote the
// child's own FP32 bound and, for a box it proved infeasible or a
// duplicate, the final state.  A child of a dropped parent has no box; for
// the others the parent's certified bound, which holds for every child box
// inside it, is folded in, and the state follows from the folded bound:
// above the incumbent, within the band below it (to the FP64 pass, which
// may prune it; below the band FP64 could not), or eligible.
__global__ void lazy_fold_kernel(const SolverCfg cfg, const SolverBufs b)
{
  const SolverDev* d = b.dev;
  if (d->done) return;
  const uint64_t total = d->n_children;
  const double gub = d->gub;
  const double floor_b = certify_floor(gub);
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = g >> cfg.log2C, r = g & ((1ULL << cfg.log2C) - 1ULL);
    const ParentInfo pi = b.pinfo[k];
    if (pi.fathom || r >= pi.nreg) {
      b.cstate[g] = kChildNone;
      continue;
    }
    const uint8_t st = b.cstate[g];
    if (st == kChildInfeasible || st == kChildDuplicate) continue;
    const double plb = b.plb[k], lb32 = b.clb[g];
    const double lb = plb > lb32 ? plb : lb32;
    b.clb[g] = lb;
    b.cstate[g] = lb > gub ? kChildDominated : lb >= floor_b ? kChildScreened : kChildEligible;
  }
}


// The screen's tallies: children bounded, and excluded by the verdicts.
__global__ void eval_count_kernel(const SolverCfg cfg, const SolverBufs b)
{
  SolverDev* d = b.dev;
  if (d->done) return;
  const uint64_t n = d->n_children;
  unsigned long long valid = 0, excluded = 0;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += (uint64_t)gridDim.x * blockDim.x) {
    const uint8_t s = b.cstate[g];
    if (s == kChildNone || s == kChildDuplicate) continue;
    ++valid;
    if (s == kChildInfeasible || s == kChildDominated) ++excluded;
  }
  unsigned long long c[2] = {valid, excluded};
  block_sum(c);
  if (threadIdx.x == 0) {
    if (c[0]) atomicAdd((unsigned long long*)&d->iter_valid, c[0]);
    if (c[1]) atomicAdd((unsigned long long*)&d->iter_excluded, c[1]);
    if (c[0] && d->use_screen) atomicAdd((unsigned long long*)&d->counters.screened_fp32, c[0]);
  }
  (void)cfg;
}

// The screen stays on while it excludes at least a quarter of the children
// it sees, and comes back on once the FP64 verdicts would have excluded a
// quarter: it never changes a decision, only whether the work is done.
__global__ void screen_policy_kernel(const SolverCfg cfg, const SolverBufs b)
{
  SolverDev* d = b.dev;
  if (d->done || cfg.precision != CMN_PRECISION_FP32_SCREEN) return;
  const uint64_t v = d->iter_valid;
  const uint64_t x = d->use_screen ? v - d->certify_count : d->iter_excluded;
  if (v > 0) d->use_screen = (x * 4 >= v) ? 1 : 0;
  d->counters.certified_fp64 += d->certify_count;
}

__device__ void size_pool(const SolverCfg& cfg, const SolverBufs& b)
{
  SolverDev* d = b.dev;
  // lazy form: the band's FP64 pass
  if (cfg.precision == CMN_PRECISION_FP32_LAZY) d->counters.certified_fp64 += d->certify_count;
  d->remaining = d->pool_size - d->n_parents;
  d->new_size = d->remaining + d->kept;
  d->free_top -= d->kept;  // taken by the appended children
  d->evict = d->new_size > cfg.cap ? 1 : 0;
  // the next iteration's parents: its E (search/driver.hpp:221-233) over the
  // pool this iteration leaves
  const uint64_t next_L = d->evict ? cfg.cap : d->new_size;
  uint64_t E = next_L < cfg.e_max ? next_L : cfg.e_max;
  const uint64_t left = cfg.iter_limit > d->expansions ? cfg.iter_limit - d->expansions : 0;
  d->pre_k = E < left ? E : left;
  d->evict_lo_key = d->pool_min_key < d->child_min_key ? d->pool_min_key : d->child_min_key;
  d->evict_hi_key = d->pool_max_key > d->child_max_key ? d->pool_max_key : d->child_max_key;
  d->pool_min_key = ~0ULL;  // refilled by the move to the other buffer
  d->pool_max_key = 0;
}

__device__ void finish_pool(const SolverCfg& cfg, const SolverBufs& b)
{
  SolverDev* d = b.dev;
  // the survivors were moved to the other buffer: exactly the cap when
  // evicting, otherwise every alive entry
  const uint64_t expect = d->evict ? cfg.cap : d->new_size;
  if (d->survivors != expect) d->error = 1;
  d->free_top += d->extent - d->survivors;  // the parents' and the evicted slots
  if (d->free_top + d->survivors != cfg.pstride) d->error = 1;
  if (d->pre_count != d->pre_k) d->error = 1;
  d->pre_valid = d->pre_k > 0 ? 1u : 0u;
  d->pool_size = d->survivors;
  d->parity = 1 - d->parity;
  if (d->dropped_min_key != ~0ULL) d->dropped_lb_min = key_to_lb(d->dropped_min_key);
  if (d->pool_size > d->counters.peak_frontier) d->counters.peak_frontier = d->pool_size;
}

// ---------------------------------------------------------------------
// the pool's rebuild, one launch
// ---------------------------------------------------------------------
// A barrier of the launch's first `blocks` blocks: each takes a ticket, the
// last one runs `last` and opens it.  The launch is cooperative, so every block is
// resident and the others wait no longer than a pass takes; the wait has a
// limit (about a second) all the same, after which the device error is set and
// false returned: the search ends there (halted).
constexpr uint32_t kBarrierSpins = 1u << 21;
template <class F>
__device__ __forceinline__ bool grid_barrier(SolverDev* d, unsigned blocks, F last)
{
  __shared__ int last_s, ok_s;
  __syncthreads();
  uint32_t gen = 0;
  if (threadIdx.x == 0) {
    gen = *(volatile uint32_t*)&d->barrier;
    __threadfence();
    last_s = atomicAdd(&d->ticket, 1u) == blocks - 1;
    __threadfence();
  }
  __syncthreads();
  if (last_s) {
    last();
    __syncthreads();
    if (threadIdx.x == 0) {
      d->ticket = 0;
      __threadfence();
      atomicAdd(&d->barrier, 1u);
      ok_s = 1;
    }
  } else if (threadIdx.x == 0) {
    int ok = 0;
    for (uint32_t i = 0; i < kBarrierSpins && !ok; ++i) ok = *(volatile uint32_t*)&d->barrier != gen;
    if (!ok) d->error = 1;
    __threadfence();
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// Blocks of a launch that take part: one per `items` of the n, so that few
// entries do not wait for the tickets of a whole GPU (n does not change while
// the kernel runs).
__device__ __forceinline__ unsigned blocks_for(uint64_t n, uint64_t items)
{
  const uint64_t want = n < 1 ? 1 : (n + items - 1) / items;
  return want < gridDim.x ? (unsigned)want : gridDim.x;
}

// Sums of two per-block counts over the blocks before this one, and over all.
__device__ __forceinline__ void blocks_before(const uint32_t* c0, const uint32_t* c1, unsigned blocks,
                                              uint64_t (&before)[2], uint64_t (&all)[2])
{
  __shared__ unsigned long long acc[4];
  __syncthreads();
  if (threadIdx.x < 4) acc[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long v[4] = {};
  for (uint32_t i = threadIdx.x; i < blocks; i += blockDim.x) {
    const uint32_t a = __ldcg(c0 + i), c = __ldcg(c1 + i);
    v[2] += a;
    v[3] += c;
    if (i < blockIdx.x) {
      v[0] += a;
      v[1] += c;
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    for (int off = 16; off > 0; off >>= 1) v[e] += __shfl_down_sync(0xffffffffu, v[e], off);
    if ((threadIdx.x & 31) == 0 && v[e]) atomicAdd(&acc[e], v[e]);
  }
  __syncthreads();
  before[0] = acc[0];
  before[1] = acc[1];
  all[0] = acc[2];
  all[1] = acc[3];
}

// ---------------------------------------------------------------------
// incumbent, prune accounting, pool finish
// ---------------------------------------------------------------------
// Counts of the children's verdicts (search/driver.hpp:319-350) and of the
// evaluations the form counts per valid child, the key range of the children
// the pool takes, and their list in order.  A count, a scan and a scatter in
// three launches took 3.5 us more of the 119 of an iteration with a few
// children.
__global__ void __launch_bounds__(kScanBlock, 2) prune_kernel(const SolverCfg cfg, const SolverBufs b)
{
  SolverDev* d = b.dev;
  if (d->done) return;
  const uint64_t n = d->n_children;
  const unsigned blocks = blocks_for(n, kScanTile);
  if (blockIdx.x >= blocks) return;
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile, per = (tiles + blocks - 1) / blocks;
  const uint64_t tile0 = (uint64_t)blockIdx.x * per < tiles ? (uint64_t)blockIdx.x * per : tiles;
  const uint64_t tile1 = tile0 + per < tiles ? tile0 + per : tiles;
  const uint64_t gub = dbits(d->gub);
  uint32_t dup = 0, inf = 0, dom = 0, kept = 0, sampled = 0, valid = 0, entries = 0;
  uint64_t mkey = ~0ULL, xkey = 0;
  for (uint64_t t = tile0; t < tile1; ++t) {
    const uint64_t t0 = tile_first(t);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
      const uint64_t g = tile_item(t0, j);
      if (g >= n) continue;
      const uint8_t s = b.cstate[g];
      if (s == kChildNone) continue;
      if (cfg.sample_all || s == kChildEligible) ++sampled;
      if (s == kChildDuplicate) {
        ++dup;
        continue;
      }
      ++valid;
      if (s == kChildInfeasible) {
        ++inf;
        continue;
      }
      const uint64_t lb = dbits(b.clb[g]);
      const bool keep = s != kChildDominated && !bits_lt(gub, lb);
      if (keep) ++kept;
      else ++dom;
      if (keep && s == kChildEligible) ++entries;  // KeptChild
      if (s == kChildEligible) {  // a superset of the kept children
        const uint64_t k = bits_key(lb);
        mkey = k < mkey ? k : mkey;
        xkey = k > xkey ? k : xkey;
      }
    }
  }
  unsigned long long c[7] = {dup, inf, dom, kept, sampled, valid, entries};
  block_sum(c);
  mkey = block_min(mkey);
  xkey = block_max(xkey);
  if (threadIdx.x == 0) {
    b.block_counts[blockIdx.x] = (uint32_t)c[6];
    if (mkey != ~0ULL) atomicMin((unsigned long long*)&d->child_min_key, (unsigned long long)mkey);
    if (xkey != 0) atomicMax((unsigned long long*)&d->child_max_key, (unsigned long long)xkey);
    if (c[0]) atomicAdd((unsigned long long*)&d->counters.pruned_duplicate, c[0]);
    if (c[1]) atomicAdd((unsigned long long*)&d->counters.pruned_infeasible, c[1]);
    if (c[2]) atomicAdd((unsigned long long*)&d->counters.pruned_dominated, c[2]);
    if (c[3]) atomicAdd((unsigned long long*)&d->counters.enqueued, c[3]);
    if (c[4]) atomicAdd((unsigned long long*)&d->counters.sampled, c[4] * cfg.S);
    if (c[5] && cfg.precision == CMN_PRECISION_FP64) atomicAdd((unsigned long long*)&d->counters.certified_fp64, c[5]);
    if (c[5] && cfg.precision == CMN_PRECISION_FP32_LAZY) atomicAdd((unsigned long long*)&d->counters.screened_fp32, c[5]);
  }
  if (!grid_barrier(d, blocks, [] {})) return;
  // the kept children's list, in order
  uint64_t base[2], all[2];
  blocks_before(b.block_counts, b.block_counts, blocks, base, all);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    d->kept = all[0];
    d->extent = d->pool_size + all[0];
  }
  const KeptChild is_kept{b};
  for (uint64_t t = tile0; t < tile1; ++t) {
    const uint64_t t0 = tile_first(t);
    bool f[kScanItems];
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
      const uint64_t g = tile_item(t0, j);
      f[j] = g < n && is_kept(g);
    }
    int rank[kScanItems];
    const int total = tile_ranks(f, rank);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j)
      if (f[j]) b.list[base[0] + (uint64_t)rank[j]] = (uint32_t)tile_item(t0, j);
    base[0] += (uint64_t)total;
    __syncthreads();  // the rank table is reused
  }
}

// Alive entries of tile `tile` inside each ranked target's threshold bucket.
__device__ __forceinline__ void eq_count(const SolverBufs& b, uint64_t tile, uint64_t n, uint32_t p,
                                         const TargetView& A, const TargetView& B, int (&c)[2])
{
  const uint64_t t0 = tile_first(tile);
  const uint64_t* __restrict__ lb = reinterpret_cast<const uint64_t*>(parity_buf(b.lb, p));
  const uint8_t* sel = parity_buf(b.sel, p);
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = tile_item(t0, j);
    if (i >= n || sel[i] != kSelAlive) continue;
    const uint64_t key = bits_key(lb[i]);
    c[0] += (A.ranked && (key & A.mask) == A.prefix) ? 1 : 0;
    c[1] += (B.ranked && (key & B.mask) == B.prefix) ? 1 : 0;
  }
}

// Marks the k smallest (key, position) entries of each target among a tile's
// alive ones: all keys below the threshold bucket, and the entries inside it
// by rank (`base`: those before the tile, advanced past it).  An entry outside
// the cap becomes kSelEvicted and is folded into the dropped floor
// (search/budget.hpp:190-209); a parent of the next iteration among those that
// stay becomes kSelNextParent.  The holes of this iteration's parents stay.
struct MarkTally {
  int stay, next;
  uint32_t viable, dominated;
  uint64_t mkey;
};
__device__ __forceinline__ void mark_tile(const SolverBufs& b, uint64_t tile, uint64_t n, uint32_t p, uint64_t gub,
                                          const TargetView& A, const TargetView& B, bool pre, uint64_t (&base)[2],
                                          MarkTally& m)
{
  const uint64_t t0 = tile_first(tile);
  const uint64_t* __restrict__ lb = reinterpret_cast<const uint64_t*>(parity_buf(b.lb, p));
  uint8_t* sel = parity_buf(b.sel, p);
  uint64_t x[kScanItems];  // raw bits of the lower bounds
  bool alive[kScanItems], eqA[kScanItems], eqB[kScanItems];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = tile_item(t0, j);
    x[j] = i < n ? lb[i] : 0;
    alive[j] = i < n && sel[i] == kSelAlive;
  }
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t key = bits_key(x[j]);
    eqA[j] = A.active && alive[j] && (key & A.mask) == A.prefix;
    eqB[j] = pre && B.active && alive[j] && (key & B.mask) == B.prefix;
  }
  int rankA[kScanItems] = {}, rankB[kScanItems] = {};
  const uint64_t baseA = base[0], baseB = base[1];
  if (A.ranked) base[0] += (uint64_t)tile_ranks<0>(eqA, rankA);  // the same for the whole grid
  if (pre && B.ranked) base[1] += (uint64_t)tile_ranks<1>(eqB, rankB);
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    if (!alive[j]) continue;
    const uint64_t key = bits_key(x[j]);
    const bool ta = A.take(key, eqA[j], baseA + (uint64_t)rankA[j]);
    const bool tb = pre && ta && B.take(key, eqB[j], baseB + (uint64_t)rankB[j]);
    const uint64_t i = tile_item(t0, j);
    if (!ta) {
      sel[i] = kSelEvicted;
      if (bits_le(x[j], gub)) {
        ++m.viable;
        m.mkey = key < m.mkey ? key : m.mkey;
      } else {
        ++m.dominated;
      }
    } else if (tb) {
      sel[i] = kSelNextParent;
    }
    m.stay += ta ? 1 : 0;
    m.next += tb ? 1 : 0;
  }
}

// Moves a tile's entries that stay, in order, to the other buffer (lower
// bound, store slot and mark), lists the store slots of the next iteration's
// parents among them in order, and pushes the store slots of the others (this
// iteration's parents and the evicted) onto the free stack in position order.
// `base`: stayers and next parents before the tile, advanced past it; `range`:
// the smallest and largest key of this thread's stayers.
__device__ __forceinline__ void copy_tile(const SolverCfg& cfg, const SolverBufs& b, uint64_t tile, uint64_t n,
                                          uint32_t p, uint64_t free_base, uint64_t (&base)[2], uint64_t (&range)[2])
{
  const uint64_t t0 = tile_first(tile);
  const uint64_t* __restrict__ slb = reinterpret_cast<const uint64_t*>(parity_buf(b.lb, p));
  const uint32_t* __restrict__ sslot = parity_buf(b.slot, p);
  const uint8_t* ssel = parity_buf(b.sel, p);
  uint64_t* __restrict__ dlb = reinterpret_cast<uint64_t*>(parity_buf(b.lb, 1 - p));
  uint32_t* __restrict__ dslot = parity_buf(b.slot, 1 - p);
  uint8_t* __restrict__ dsel = parity_buf(b.sel, 1 - p);
  bool f[kScanItems], g[kScanItems], in[kScanItems];
  uint64_t x[kScanItems];  // raw bits of the lower bounds
  uint32_t sl[kScanItems];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    const uint64_t i = tile_item(t0, j);
    in[j] = i < n;
    const uint8_t sv = in[j] ? ssel[i] : kSelParent;
    x[j] = in[j] ? slb[i] : 0;
    sl[j] = in[j] ? sslot[i] : 0u;
    f[j] = sv == kSelAlive || sv == kSelNextParent;
    g[j] = sv == kSelNextParent;
  }
#pragma unroll
  for (int j = 0; j < kScanItems; ++j)
    if (f[j]) {
      const uint64_t k = bits_key(x[j]);
      range[0] = k < range[0] ? k : range[0];
      range[1] = k > range[1] ? k : range[1];
    }
  int rank[kScanItems], prank[kScanItems], total[2];  // stayers / next parents before each item
  tile_ranks2(f, g, rank, prank, total);
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    if (!in[j]) continue;
    const uint64_t i = tile_item(t0, j);
    const uint64_t stay_before = base[0] + (uint64_t)rank[j];
    if (f[j]) {
      dlb[stay_before] = x[j];
      dslot[stay_before] = sl[j];
      dsel[stay_before] = g[j] ? kSelParent : kSelAlive;
      if (g[j]) {
        const uint64_t pos = base[1] + (uint64_t)prank[j];
        if (pos < cfg.e_max) b.pslot[pos] = sl[j];
        else b.dev->error = 1;
      }
    } else {
      b.free_slots[free_base + (i - stay_before)] = sl[j];
    }
  }
  base[0] += (uint64_t)total[0];
  base[1] += (uint64_t)total[1];
}

// Sizes, the radix passes, the marks, the move and the staging of the next
// iteration's parents: each needs all of the one before, so the blocks meet at
// a barrier between them, five and one per radix pass (a small pool's keys
// differ in two or three digits).  Each block keeps the same consecutive
// tiles throughout, so it needs only the counts of the blocks before it and no
// scan of its own.  As twelve launches over a grid of every tile the pool
// could have, an iteration of the n = 4 plain solve (a few hundred entries,
// room for 2^24) spent 76 of its 178 us here; the one launch takes 23.
__global__ void __launch_bounds__(kScanBlock, 2) rebuild_kernel(const SolverCfg cfg, const SolverBufs b)
{
  SolverDev* d = b.dev;
  if (halted(*d)) return;
  const uint64_t n = d->extent;
  const unsigned blocks = blocks_for(n, kScanBlock);
  if (blockIdx.x >= blocks) return;
  // (1) sizes, the select's start
  if (!grid_barrier(d, blocks, [&] {
        if (threadIdx.x == 0) size_pool(cfg, b);
        __syncthreads();
        radix_init(cfg, b);
      }))
    return;
  const uint64_t pre_k = d->pre_k, free_base = d->free_top;
  const uint32_t p = d->parity;
  // (2) digits of up to 11 bits from below the keys' common leading bits
  for (int pass = 0; pass < (64 + kRadixBits - 1) / kRadixBits; ++pass) {
    bool go[2];
    if (!radix_hist(b, blocks, n, p, go)) break;  // the same for every block
    if (!grid_barrier(d, blocks, [&] {
          for (int t = 0; t < 2; ++t)
            if (go[t]) radix_pick(b, b.radix + t);
        }))
      return;
  }
  const TargetView A(b.radix[0]), B(b.radix[1]);
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile, per = (tiles + blocks - 1) / blocks;
  const uint64_t tile0 = (uint64_t)blockIdx.x * per < tiles ? (uint64_t)blockIdx.x * per : tiles;
  const uint64_t tile1 = tile0 + per < tiles ? tile0 + per : tiles;
  uint64_t base[2] = {0, 0}, all[2];
  // (3) ranks inside the threshold buckets, where one is split
  if (A.ranked || B.ranked) {
    int c[2] = {0, 0};
    for (uint64_t t = tile0; t < tile1; ++t) eq_count(b, t, n, p, A, B, c);
    const int c0 = tile_count<0>(c[0]), c1 = tile_count<1>(c[1]);
    if (threadIdx.x == 0) {
      b.block_counts[blockIdx.x] = (uint32_t)c0;
      b.block_counts2[blockIdx.x] = (uint32_t)c1;
    }
    if (!grid_barrier(d, blocks, [] {})) return;
    blocks_before(b.block_counts, b.block_counts2, blocks, base, all);
  }
  // (4) the marks
  MarkTally m = {0, 0, 0, 0, ~0ULL};
  {
    const uint64_t gub = dbits(d->gub);
    for (uint64_t t = tile0; t < tile1; ++t) {
      mark_tile(b, t, n, p, gub, A, B, pre_k > 0, base, m);
      __syncthreads();  // the rank tables are reused
    }
    unsigned long long v[4] = {(unsigned)m.stay, (unsigned)m.next, m.viable, m.dominated};
    block_sum(v);
    const uint64_t mk = block_min(m.mkey);
    if (threadIdx.x == 0) {
      b.block_offsets[blockIdx.x] = (uint32_t)v[0];
      b.block_offsets2[blockIdx.x] = (uint32_t)v[1];
      if (v[2]) atomicAdd((unsigned long long*)&d->counters.dropped_viable, v[2]);
      if (v[3]) atomicAdd((unsigned long long*)&d->counters.dropped_dominated, v[3]);
      if (mk != ~0ULL) atomicMin((unsigned long long*)&d->dropped_min_key, (unsigned long long)mk);
    }
  }
  if (!grid_barrier(d, blocks, [] {})) return;
  // (5) the move, the key range of what stays
  blocks_before(b.block_offsets, b.block_offsets2, blocks, base, all);
  uint64_t range[2] = {~0ULL, 0};
  for (uint64_t t = tile0; t < tile1; ++t) {
    copy_tile(cfg, b, t, n, p, free_base, base, range);
    __syncthreads();
  }
  range[0] = block_min(range[0]);
  range[1] = block_max(range[1]);
  if (threadIdx.x == 0) {
    if (range[0] != ~0ULL) atomicMin((unsigned long long*)&d->pool_min_key, (unsigned long long)range[0]);
    if (range[1] != 0) atomicMax((unsigned long long*)&d->pool_max_key, (unsigned long long)range[1]);
  }
  // (6) the next parents' boxes; one thread closes the iteration
  if (!grid_barrier(d, blocks, [] {})) return;
  const uint64_t next = all[1] < cfg.e_max ? all[1] : cfg.e_max;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    d->survivors = all[0];
    d->pre_count = all[1];
    finish_pool(cfg, b);
  }
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < next; k += (uint64_t)blocks * blockDim.x)
    stage_parent(cfg, b, __ldcg(b.pslot + k), k);
  if (threadIdx.x == 0) stamp_last(d->stamps + 4, (uint64_t)blockIdx.x * blockDim.x < next);
}

__global__ void pool_min_kernel(const SolverBufs b, uint64_t* viable_out)
{
  SolverDev* d = b.dev;
  const uint64_t n = d->pool_size;
  const double* lb = parity_buf(b.lb, d->parity);
  const double gub = d->gub;
  uint64_t mkey = ~0ULL;
  unsigned long long viable = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = lb_key(lb[i]);
    mkey = k < mkey ? k : mkey;
    if (lb[i] <= gub) ++viable;
  }
  unsigned long long c[1] = {viable};
  block_sum(c);
  mkey = block_min(mkey);
  if (threadIdx.x == 0) {
    if (mkey != ~0ULL) atomicMin((unsigned long long*)&d->pool_min_key, (unsigned long long)mkey);
    if (viable_out && c[0]) atomicAdd((unsigned long long*)viable_out, c[0]);
  }
}

__global__ void pool_min_reset_kernel(const SolverBufs b, uint64_t* viable_out)
{
  b.dev->pool_min_key = ~0ULL;
  if (viable_out) *viable_out = 0;
}

// ---------------------------------------------------------------------
// host: enqueue one iteration
// ---------------------------------------------------------------------
static int tiles(uint64_t max_items) { return (int)((max_items + kScanTile - 1) / kScanTile); }

static void scan(const SolverBufs& b, const uint64_t* n_items_dev, uint64_t* total_dev, cudaStream_t s)
{
  scan_kernel<<<1, 1024, 0, s>>>(b.block_counts, b.block_offsets, n_items_dev, total_dev, &b.dev->done);
}

template <class P>
static void compact(const P& pred, uint64_t max_items, const uint64_t* n_items_dev, uint64_t* total_dev,
                    const SolverBufs& b, cudaStream_t s)
{
  count_kernel<P><<<tiles(max_items), kScanBlock, 0, s>>>(pred, b.block_counts);
  scan(b, n_items_dev, total_dev, s);
}

template <class P, class Op>
static void scatter(const P& pred, const Op& op, uint64_t max_items, cudaStream_t s, const SolverBufs& b)
{
  scatter_kernel<P, Op><<<tiles(max_items), kScanBlock, 0, s>>>(pred, op, b.block_offsets);
}

// A kernel whose blocks meet at barriers, over the tiles of max_items: as many
// blocks as are resident at once, no more than the tiles.
static cudaError_t cooperative(void (*kernel)(SolverCfg, SolverBufs), uint64_t max_items, const SolverCfg& cfg,
                               const SolverBufs& b, cudaStream_t s)
{
  int occ = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kScanBlock, 0);
  if (e != cudaSuccess) return e;
  const int grid = std::min(tiles(max_items), sm_count() * std::min(occ, 2));
  void* args[] = {const_cast<SolverCfg*>(&cfg), const_cast<SolverBufs*>(&b)};
  return cudaLaunchCooperativeKernel((const void*)kernel, dim3((unsigned)grid), dim3(kScanBlock), args, 0, s);
}

cudaError_t solver_iteration(const SolverCfg& cfg, const SolverBufs& b, int eval_grid, int sample_grid,
                             cudaStream_t s, const SideStream& side)
{
  const bool lazy = cfg.precision == CMN_PRECISION_FP32_LAZY;
  const uint64_t max_children = cfg.e_max << cfg.log2C;
  begin_kernel<<<1, 1, 0, s>>>(cfg, b);

  // (1b) lazy form: the FP64 verdict of every staged parent -- its bound
  // has been an FP32 one (with its own parent's FP64 bound folded in) since
  // it was appended.  It runs on the side stream, beside the branching and
  // the FP32 child bounds, which do not read it: the 2^-B share of boxes
  // it evaluates leaves part of the GPU idle on its own.
  if (lazy) {
    cudaError_t e = cudaEventRecord(side.fork, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side.stream, side.fork, 0);
    if (e != cudaSuccess) return e;
    EvalArgs pa = {};
    pa.prog = b.prog64;
    pa.prog_len = cfg.prog_len;
    pa.n_vars = cfg.n_vars;
    pa.n_slots = cfg.n_slots;
    pa.log2C = 0;  // one "child" per parent: the parent box itself
    pa.plo = b.plo;
    pa.phi = b.phi;
    pa.pstride = cfg.e_max;
    pa.n_children_dev = &b.dev->n_parents;
    pa.done = &b.dev->done;
    pa.out_lb = b.plb;
    pa.out_flag = b.pfeas;
    pa.sched = b.sched;
    pa.g_max = cfg.g_max;
    pa.capacity = cfg.eval_capacity;
    pa.error = &b.dev->error;
    pa.chain = b.chain;
    pa.max_boxes = cfg.e_max;
    pa.t_first = b.dev->stamps + 5;
    pa.t_last = b.dev->stamps + 6;
    e = launch_eval(pa, 6, false, eval_grid, kEvalThreads, side.stream);
    if (e != cudaSuccess) return e;
    e = cudaEventRecord(side.join, side.stream);
    if (e != cudaSuccess) return e;
  }

  // (2) branch
  {
    const int grid = (int)std::min<uint64_t>((cfg.e_max + 127) / 128, 2048);
    if (cfg.n_vars <= 8) branch_kernel<8><<<grid, 128, 0, s>>>(cfg, b);
    else if (cfg.n_vars <= 32) branch_kernel<32><<<grid, 128, 0, s>>>(cfg, b);
    else if (cfg.n_vars <= kPolicyLocal) branch_kernel<kPolicyLocal><<<grid, 128, 0, s>>>(cfg, b);
    else branch_kernel<0><<<grid, 128, 0, s>>>(cfg, b);
  }

  // (3) bound every child: FP64, or FP32 screen + FP64 certify
  EvalArgs ea = {};
  ea.n_vars = cfg.n_vars;
  ea.n_slots = cfg.n_slots;
  ea.log2C = cfg.log2C;
  ea.plo = b.plo;
  ea.phi = b.phi;
  ea.pstride = cfg.e_max;
  ea.pinfo = b.pinfo;
  ea.slots = b.slots;
  ea.max_slots = cfg.max_slots;
  ea.n_children_dev = &b.dev->n_children;
  ea.gub = &b.dev->gub;
  ea.done = &b.dev->done;
  ea.out_lb = b.clb;
  ea.out_flag = b.cstate;
  ea.error = &b.dev->error;
  ea.prog_len = cfg.prog_len;
  ea.sched = b.sched;
  ea.g_max = cfg.g_max;
  ea.capacity = cfg.eval_capacity;
  ea.chain = b.chain;  // read by the FP64 passes
  ea.max_boxes = max_children;
  cudaError_t e;
  if (cfg.precision == CMN_PRECISION_FP32_SCREEN) {
    ea.prog = b.prog32;
    ea.plo32 = b.plo32;
    ea.phi32 = b.phi32;
    ea.use_screen = &b.dev->use_screen;
    e = launch_eval(ea, 2, true, eval_grid, kEvalThreads, s);
    if (e != cudaSuccess) return e;
    ScreenedChild sc{b};
    compact(sc, max_children, &b.dev->n_children, &b.dev->certify_count, b, s);
    scatter(sc, ListChild{b}, max_children, s, b);
    EvalArgs ca = ea;
    ca.prog = b.prog64;
    ca.plo32 = nullptr;
    ca.phi32 = nullptr;
    ca.list = b.list;
    ca.list_count = &b.dev->certify_count;
    e = launch_eval(ca, 3, false, eval_grid, kEvalThreads, s);
    if (e != cudaSuccess) return e;
  } else if (lazy) {
    ea.prog = b.prog32;
    ea.plo32 = b.plo32;
    ea.phi32 = b.phi32;
    ea.parent_lb = nullptr;  // folded in by lazy_fold_kernel
    ea.t_last = b.dev->stamps + 7;
    if (cfg.inc_tile) {
      ea.n_parents_dev = &b.dev->n_parents;
      e = launch_lazy_children(ea, cfg.e_max, s);
    } else if (cfg.inc) {
      ea.inc_segments = cfg.inc_segments;
      ea.n_parents_dev = &b.dev->n_parents;
      ea.inc_seg = b.inc_seg;
      ea.inc_off = b.inc_off;
      ea.inc_pcs = b.inc_pcs;
      ea.inc_common = b.inc_common;
      ea.inc_parts = b.inc_parts;
      e = launch_inc(ea, eval_grid, kEvalThreads, s);
    } else {
      e = launch_eval(ea, 5, true, eval_grid, kEvalThreads, s);
    }
    if (e != cudaSuccess) return e;
    // join the parents' FP64 verdict: drop the boxes it excludes, fold the
    // certified bounds into their children
    e = cudaStreamWaitEvent(s, side.join, 0);
    if (e != cudaSuccess) return e;
    {
      const int pgrid = (int)std::min<uint64_t>((cfg.e_max + 255) / 256, 1024);
      lazy_drop_kernel<<<pgrid, 256, 0, s>>>(cfg, b);
      const int cgrid = (int)std::min<uint64_t>((max_children + 255) / 256, 2048);
      lazy_fold_kernel<<<cgrid, 256, 0, s>>>(cfg, b);
    }
    // the survivors within the band below the incumbent, in FP64
    ScreenedChild sc{b};
    compact(sc, max_children, &b.dev->n_children, &b.dev->certify_count, b, s);
    scatter(sc, ListChild{b}, max_children, s, b);
    EvalArgs ca = ea;
    ca.prog = b.prog64;
    ca.plo32 = nullptr;
    ca.phi32 = nullptr;
    ca.parent_lb = b.plb;
    ca.t_last = nullptr;
    ca.inc_segments = 0;
    ca.list = b.list;
    ca.list_count = &b.dev->certify_count;
    e = launch_eval(ca, 3, false, eval_grid, kEvalThreads, s);
    if (e != cudaSuccess) return e;
  } else {
    ea.prog = b.prog64;
    e = launch_eval(ea, 1, false, eval_grid, kEvalThreads, s);
    if (e != cudaSuccess) return e;
  }
  if (cfg.precision == CMN_PRECISION_FP32_SCREEN) {
    const int grid = (int)std::min<uint64_t>((max_children + 255) / 256, 1024);
    eval_count_kernel<<<grid, 256, 0, s>>>(cfg, b);
    screen_policy_kernel<<<1, 1, 0, s>>>(cfg, b);
  }

  // (4) sample, ArgMin, incumbent update and witness
  SampleArgs sa = {};
  sa.prog = b.prog64;
  sa.prog_len = cfg.prog_len;
  sa.n_vars = cfg.n_vars;
  sa.n_slots = cfg.n_slots;
  sa.log2C = cfg.log2C;
  sa.plo = b.plo;
  sa.phi = b.phi;
  sa.pstride = cfg.e_max;
  sa.pinfo = b.pinfo;
  sa.slots = b.slots;
  sa.max_slots = cfg.max_slots;
  sa.var_kinds = b.kinds;
  sa.root_lb = b.root_lb;
  sa.root_ub = b.root_ub;
  sa.n_children_dev = &b.dev->n_children;
  sa.S = cfg.S;
  sa.salt_base_dev = &b.dev->salt_base;
  sa.sample_all = cfg.sample_all;
  sa.state = b.cstate;
  sa.gub = &b.dev->gub;
  sa.done = &b.dev->done;
  sa.block_best = b.block_best;
  sa.rejected = (unsigned long long*)&b.dev->counters.witness_rejected;
  sa.sched = b.sched;
  sa.g_max = cfg.g_max;
  sa.capacity = cfg.sample_capacity;
  sa.lg_min = cfg.sample_lg_min;
  sa.chain = b.chain;
  sa.t_first = b.dev->stamps + 2;
  if (cfg.precision == CMN_PRECISION_FP32_LAZY) {
    // FP32 screen of every sample, then each chunk's best in FP64
    SampleArgs qa = sa;
    qa.lg_min = cfg.screen_lg_min;
    qa.prog = b.prog32p;
    qa.cbest = b.cbest;
    e = chain_screen_fits(qa) ? launch_chain_screen(qa, max_children, s)
                              : launch_sample_screen(qa, cfg.screen_grid, kEvalThreads, s);
    if (e != cudaSuccess) return e;
    sa.cbest = b.cbest;
    sa.t_first = nullptr;
  }
  e = launch_sample(sa, sample_grid, kEvalThreads, s);
  if (e != cudaSuccess) return e;
  Cand* best = b.block_best + b.n_block_best - 1;  // last entry holds the result
  const WitnessArgs w = {b.plo, b.phi, cfg.e_max, b.pinfo, b.slots, cfg.max_slots, b.kinds, cfg.n_vars, cfg.S, 0,
                         &b.dev->salt_base, 0, b.best_point};
  e = launch_candidate(b.block_best, sample_grid, best, w,
                       Incumbent{&b.dev->done, &b.dev->gub, &b.dev->best, &b.dev->have_best, &b.dev->improved, b.dev->stamps + 3}, s);
  if (e != cudaSuccess) return e;

  // (5) prune with the new incumbent and rebuild the pool
  // (the kept children go behind the pool in the current buffer; the parents
  // stay there as holes until the one compaction below)
  e = cooperative(prune_kernel, max_children, cfg, b, s);
  if (e != cudaSuccess) return e;
  {
    const int grid = (int)std::min<uint64_t>((max_children + 255) / 256, 4096);
    if (cfg.n_vars > 16) append_boxes_kernel<32><<<grid, 256, 0, s>>>(cfg, b);
    else if (cfg.n_vars > 8) append_boxes_kernel<16><<<grid, 256, 0, s>>>(cfg, b);
    else append_children_kernel<<<grid, 256, 0, s>>>(cfg, b);
  }

  // (6) over the cap: keep the `cap` best alive entries, fold the rest into
  // the floor; select and stage the next iteration's parents; move every alive
  // entry to the other buffer in order
  e = cooperative(rebuild_kernel, cfg.pstride, cfg, b, s);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t solver_init(const SolverCfg& cfg, const SolverBufs& b, const double* root_lb_dev,
                        const double* root_ub_dev, double gub0, cudaStream_t s)
{
  const int grid = (int)std::min<uint64_t>((cfg.pstride + 255) / 256, 4096);
  free_init_kernel<<<grid, 256, 0, s>>>(cfg, b);
  cudaMemsetAsync(b.sel[0], kSelAlive, cfg.pstride, s);
  init_kernel<<<1, 256, 0, s>>>(cfg, b, root_lb_dev, root_ub_dev, gub0);
  cudaMemsetAsync(b.sel[1], kSelAlive, cfg.pstride, s);
  return cudaGetLastError();
}

cudaError_t solver_frontier_gather(const SolverCfg& cfg, const SolverBufs& b, uint64_t start, uint64_t count,
                                   double* boxes, uint32_t* depths, cudaStream_t s)
{
  if (count == 0) return cudaSuccess;
  const int grid = (int)std::min<uint64_t>((count + 255) / 256, 4096);
  frontier_gather_kernel<<<grid, 256, 0, s>>>(cfg, b, start, count, boxes, depths);
  return cudaGetLastError();
}

cudaError_t solver_pool_stats(const SolverCfg& cfg, const SolverBufs& b, uint64_t* viable_dev, cudaStream_t s)
{
  pool_min_reset_kernel<<<1, 1, 0, s>>>(b, viable_dev);
  const int grid = (int)std::min<uint64_t>((cfg.pstride + 255) / 256, 4096);
  pool_min_kernel<<<grid, 256, 0, s>>>(b, viable_dev);
  return cudaGetLastError();
}

}  // namespace cmn
