// batch_chain_kernels.cu -- the tile kernels (chain_tiles.cuh,
// chain32_tiles.cuh, point_tiles.cuh) over many instances: one launch walks
// the tiles of every instance whose program is a set of sum chains, longest
// program first (batch_live_kernel lays the tiles out).
//
// Each tile is one instance's, so a block or warp that draws it looks the
// instance up once and runs the single-instance code on that instance's
// slices of the batch's arrays.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "batch.hpp"
#include "chain32_tiles.cuh"
#include "chain_tiles.cuh"
#include "launch.hpp"
#include "point_tiles.cuh"

namespace cmn {

namespace {

// Instance `slot`'s slices, as the single-instance kernels take them.
__device__ __forceinline__ void slot_args(const BatchCfg& c, const BatchBufs& b, uint64_t slot, EvalArgs& a)
{
  const InstDesc& d = b.desc[slot];
  const InstState& st = b.st[slot];
  a = {};  // what is not set below is off
  a.prog = d.prog64;
  a.prog_len = d.prog_len;
  a.n_vars = d.n_vars;
  a.log2C = c.log2C;
  a.plo = b.plo + splane(c, slot, 0);
  a.phi = b.phi + splane(c, slot, 0);
  a.plo32 = b.plo32 != nullptr ? b.plo32 + splane(c, slot, 0) : nullptr;
  a.phi32 = b.phi32 != nullptr ? b.phi32 + splane(c, slot, 0) : nullptr;
  a.pstride = c.e_max;
  a.pinfo = b.pinfo + slot * c.e_max;
  a.slots = b.slots + slot * c.e_max * c.max_slots;
  a.max_slots = c.max_slots;
  a.n_children = st.n_parents << c.log2C;
  a.n_parents_dev = &st.n_parents;
  a.gub = &st.gub;
  a.out_lb = b.clb + slot * c.child_stride;
  a.out_flag = b.cstate + slot * c.child_stride;
  a.chain = d.chain;
}

__device__ __forceinline__ void point_args(const BatchCfg& c, const BatchBufs& b, uint64_t slot, SampleArgs& a)
{
  const InstDesc& d = b.desc[slot];
  const InstState& st = b.st[slot];
  a = {};  // what is not set below is off
  a.prog = d.prog64;
  a.prog_len = d.prog_len;
  a.n_vars = d.n_vars;
  a.log2C = c.log2C;
  a.plo = b.plo + splane(c, slot, 0);
  a.phi = b.phi + splane(c, slot, 0);
  a.pstride = c.e_max;
  a.pinfo = b.pinfo + slot * c.e_max;
  a.slots = b.slots + slot * c.e_max * c.max_slots;
  a.max_slots = c.max_slots;
  a.var_kinds = d.kinds;
  a.root_lb = d.root_lb;
  a.root_ub = d.root_ub;
  a.S = c.S;
  a.salt_base_dev = &st.salt_base;
  a.sample_all = c.sample_all;
  a.state = b.cstate + slot * c.child_stride;
  a.sched = d.sched;
  a.cbest = c.precision == CMN_PRECISION_FP32_LAZY ? b.cbest + slot * c.child_stride : nullptr;
  a.chain = d.chain;
}

}  // namespace

// Constraints: kFused the staged parents (pfeas), otherwise the children
// (cstate).
template <int kMode, bool kFused>
__global__ void __launch_bounds__(kTileWarps * 32, 4) batch_constraints_kernel(const BatchCfg c, const BatchBufs b)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TileShared sh;
  __shared__ EvalArgs a;
  __shared__ uint64_t first_s;
  const uint64_t* base = kFused ? b.ptile : b.ctile;
  const int log_boxes = (int)b.live[kFused ? 1 : 2];
  const uint64_t tiles = base[c.K];
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (threadIdx.x == 0) {
      const uint64_t pos = position_of(base, c.K, tile), slot = b.order[pos];
      first_s = base[pos];
      slot_args(c, b, slot, a);
      if (kFused) {  // one "child" per parent: the parent box itself
        a.log2C = 0;
        a.pinfo = nullptr;
        a.n_children = b.st[slot].n_parents;
        a.out_flag = b.pfeas + slot * c.e_max;
      }
    }
    __syncthreads();
    constraints_tile<kMode, kFused>(a, smem_raw, sh, log_boxes, tile - first_s, a.n_children);
  }
}

// The plain form's objectives, a warp per 32 children.
__global__ void __launch_bounds__(kObjThreads, 5) batch_siblings_kernel(const BatchCfg c, const BatchBufs b, int families)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  unsigned char* smem = smem_raw + family_bytes(families, c.max_slots, false) * wid;
  const uint64_t tiles = b.stile[c.K];
  for (uint64_t tile = (uint64_t)blockIdx.x * W + wid; tile < tiles; tile += (uint64_t)gridDim.x * W) {
    const uint64_t pos = position_of(b.stile, c.K, tile);
    EvalArgs a;
    slot_args(c, b, b.order[pos], a);
    siblings_tile<1, false>(a, smem, 1, families, tile - b.stile[pos], a.n_children);
  }
}

// The lazy form's child bounds, the parents' certified bounds folded in.
__global__ void __launch_bounds__(kLazyThreads, 2) batch_lazy_kernel(const BatchCfg c, const BatchBufs b)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LazyShared sh;
  __shared__ EvalArgs a;
  __shared__ uint64_t first_s;
  const uint64_t tiles = b.ltile[c.K];
  const LazyShape h = {c.lazy_chains, c.lazy_parts};
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (threadIdx.x == 0) {
      const uint64_t pos = position_of(b.ltile, c.K, tile), slot = b.order[pos];
      first_s = b.ltile[pos];
      slot_args(c, b, slot, a);
      a.prog = b.desc[slot].prog32;
      a.parent_lb = b.plb + slot * c.e_max;
    }
    __syncthreads();
    lazy_tile(a, h, smem_raw, sh, tile - first_s, *a.n_parents_dev);
  }
}

// Points of every sampled child: the lazy form's FP32 screen (cbest), or the
// plain form's samples (cval, ce: a child's best FP64 value, +inf where none
// is better than the incumbent or its tile's best).
template <bool kScreen>
__global__ void __launch_bounds__(kPointThreads) batch_points_kernel(const BatchCfg c, const BatchBufs b)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint8_t list_s[kPointThreads];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  uint8_t* list = list_s + wid * 32;
  const int pts = 1 << c.log_pts;
  stamp_first(b.stamps + 2);
  const uint64_t tiles = b.qtile[c.K];
  for (uint64_t tile = (uint64_t)blockIdx.x * W + wid; tile < tiles; tile += (uint64_t)gridDim.x * W) {
    const uint64_t pos = position_of(b.qtile, c.K, tile), slot = b.order[pos];
    const uint64_t w0 = tile - b.qtile[pos], total = b.st[slot].n_parents << c.log2C;
    SampleArgs a;
    point_args(c, b, slot, a);
    const uint64_t salt_base = b.st[slot].salt_base;
    if (kScreen) {
      float* x = reinterpret_cast<float*>(smem_raw + wid * point_bytes(c.n_max + 1, c.log_pts));
      screen_tile(a, x, list, c.log_pts, w0, total, salt_base);
      continue;
    }
    double* x64 = reinterpret_cast<double*>(smem_raw) + (size_t)wid * c.n_max;
    float* x32 = reinterpret_cast<float*>(smem_raw + (size_t)W * c.n_max * 8 + wid * point_bytes(c.n_max, c.log_pts));
    const uint64_t g = (w0 << c.log_pts) + lane, cbase = slot * c.child_stride;
    const bool mine = lane < pts && g < total;
    if (mine) b.cval[cbase + g] = INFINITY;
    PointOf p = {};
    const bool take = mine && point_child(a, g, salt_base, p);
    const double gub = b.st[slot].gub;
    unsigned long long rejected = 0;
    for (uint64_t i = 0; i < c.S; ++i) {
      p.i = i;
      __syncwarp();
      sample_tile(a, x64, x32, list, c.log_pts, p, take && (!p.fathom || i == 0), b.sbest + slot, gub, rejected,
                  [&](const PointOf& o, double value) {
                    const uint64_t at = cbase + (o.k << c.log2C) + o.r;
                    if (value < b.cval[at]) {  // samples come in order: a tie keeps the first
                      b.cval[at] = value;
                      b.ce[at] = o.r * (o.fathom ? 1 : c.S) + o.i;
                    }
                  });
    }
    if (rejected) atomicAdd((unsigned long long*)&b.st[slot].counters.witness_rejected, rejected);
  }
}

// The lazy form's picks, one per chunk of 32 children, in FP64 (cval, ce; the
// chunk's other children +inf): a warp per 2^kLogPicks
// chunks of an instance (few, so that the picks that need FP64, one after the
// other in a warp, spread over the SMs).
constexpr int kLogPicks = 3;

__global__ void __launch_bounds__(kPointThreads) batch_picks_kernel(const BatchCfg c, const BatchBufs b)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint8_t list_s[kPointThreads];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  double* x64 = reinterpret_cast<double*>(smem_raw) + (size_t)wid * c.n_max;
  float* x32 = reinterpret_cast<float*>(smem_raw + (size_t)W * c.n_max * 8 + wid * point_bytes(c.n_max, c.log_pts));
  const int log_pts = c.log_pts < kLogPicks ? c.log_pts : kLogPicks, pts = 1 << log_pts;
  const uint64_t per_slot = (((c.child_stride + 31) >> 5) + pts - 1) >> log_pts;
  for (uint64_t w = (uint64_t)blockIdx.x * W + wid; w < c.K * per_slot; w += (uint64_t)gridDim.x * W) {
    const uint64_t pos = w / per_slot, slot = b.order[pos];
    const uint64_t total = b.st[slot].n_parents << c.log2C, chunk = ((w - pos * per_slot) << log_pts) + lane;
    if (((w - pos * per_slot) << (log_pts + 5)) >= total || !b.desc[slot].tile || !b.desc[slot].chain.points) continue;
    SampleArgs a;
    point_args(c, b, slot, a);
    const uint64_t cbase = slot * c.child_stride;
    PointOf p = {};
    bool cand = lane < pts && (chunk << 5) < total;
    if (cand) {
      const uint64_t g1 = total < (chunk << 5) + 32 ? total : (chunk << 5) + 32;
      for (uint64_t g = chunk << 5; g < g1; ++g) b.cval[cbase + g] = INFINITY;
      cand = chunk_point(a, chunk, total, b.st[slot].salt_base, p);
    }
    __syncwarp();
    unsigned long long rejected = 0;
    sample_tile(a, x64, x32, list_s + wid * 32, log_pts, p, cand, b.sbest + slot, b.st[slot].gub, rejected,
                [&](const PointOf& o, double value) {
                  const uint64_t at = cbase + (o.k << c.log2C) + o.r;
                  b.cval[at] = value;
                  b.ce[at] = o.r * (o.fathom ? 1 : c.S) + o.i;
                });
    if (rejected) atomicAdd((unsigned long long*)&b.st[slot].counters.witness_rejected, rejected);
  }
}

// ---- host ----
static size_t constraints_smem(const BatchCfg& c) { return tile_smem_bytes(c.n_max, c.max_slots, 32); }
static int families_of(const BatchCfg& c) { return 32 >> (c.log2C < 5 ? c.log2C : 5); }
static size_t siblings_smem(const BatchCfg& c) { return (kObjThreads / 32) * family_bytes(families_of(c), c.max_slots, false); }
static size_t lazy_bytes(const BatchCfg& c)
{
  return lazy_smem(c.n_max, c.max_slots, LazyShape{c.lazy_chains, c.lazy_parts}, 1 << c.log2C);
}
static size_t points_smem(const BatchCfg& c, bool screen)
{
  return (size_t)(kPointThreads / 32) *
         (screen ? point_bytes(c.n_max + 1, c.log_pts) : (size_t)c.n_max * 8 + point_bytes(c.n_max, c.log_pts));
}
static size_t picks_smem(const BatchCfg& c) { return points_smem(c, false); }

void batch_tile_config(BatchCfg& c, int max_smem)
{
  const size_t room = (size_t)max_smem - 2048;
  const bool lazy = c.precision == CMN_PRECISION_FP32_LAZY;
  c.sms = sm_count();
  c.log_pts = log_points(c.n_max + 1);
  c.tiles = c.precision != CMN_PRECISION_FP32_SCREEN && constraints_smem(c) <= room && points_smem(c, true) <= room &&
            picks_smem(c) <= room;
  if (lazy) {
    c.lazy_parts = (1 << c.log2C) + 1;
    c.lazy_chains = c.max_slots <= kLazySlots ? c.seg_max : 0;
    while (c.lazy_chains > 4 && lazy_bytes(c) > room / 2) c.lazy_chains = (c.lazy_chains + 1) / 2;
    if (c.lazy_chains < 1 || lazy_bytes(c) > room) c.tiles = 0;
  } else {
    if (c.log2C < 1 || siblings_smem(c) > room) c.tiles = 0;
  }
}

bool batch_tile_takes(const BatchCfg& c, const ChainTab& t)
{
  if (!c.tiles || t.n_seg == 0 || !t.pure_objective) return false;
  return c.precision == CMN_PRECISION_FP32_LAZY ? t.term32 != nullptr && t.term_pt != nullptr : t.points != 0;
}

BatchTileGrids batch_tile_grids(const BatchCfg& c)
{
  BatchTileGrids g;
  if (!c.tiles) return g;
  if (c.precision == CMN_PRECISION_FP32_LAZY) {
    g.constraints = (int)resident_blocks(~0ULL, batch_constraints_kernel<0, true>, kTileWarps * 32, constraints_smem(c));
    g.lazy = (int)resident_blocks(~0ULL, batch_lazy_kernel, kLazyThreads, lazy_bytes(c));
    g.points = (int)resident_blocks(~0ULL, batch_points_kernel<true>, kPointThreads, points_smem(c, true));
    g.picks = (int)resident_blocks(~0ULL, batch_picks_kernel, kPointThreads, picks_smem(c));
  } else {
    g.children = (int)resident_blocks(~0ULL, batch_constraints_kernel<1, false>, kTileWarps * 32, constraints_smem(c));
    g.objective = (int)resident_blocks(~0ULL, batch_siblings_kernel, kObjThreads, siblings_smem(c));
    g.points = (int)resident_blocks(~0ULL, batch_points_kernel<false>, kPointThreads, points_smem(c, false));
  }
  return g;
}

cudaError_t batch_tile_parents(const BatchCfg& c, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s)
{
  if (!c.tiles) return cudaSuccess;
  batch_constraints_kernel<0, true><<<g.constraints, kTileWarps * 32, constraints_smem(c), s>>>(c, b);
  return cudaGetLastError();
}

cudaError_t batch_tile_lazy(const BatchCfg& c, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s)
{
  if (!c.tiles) return cudaSuccess;
  batch_lazy_kernel<<<g.lazy, kLazyThreads, lazy_bytes(c), s>>>(c, b);
  return cudaGetLastError();
}

cudaError_t batch_tile_children(const BatchCfg& c, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s)
{
  if (!c.tiles) return cudaSuccess;
  batch_constraints_kernel<1, false><<<g.children, kTileWarps * 32, constraints_smem(c), s>>>(c, b);
  batch_siblings_kernel<<<g.objective, kObjThreads, siblings_smem(c), s>>>(c, b, families_of(c));
  return cudaGetLastError();
}

cudaError_t batch_tile_points(const BatchCfg& c, const BatchBufs& b, const BatchTileGrids& g, cudaStream_t s)
{
  if (!c.tiles) return cudaSuccess;
  if (c.precision == CMN_PRECISION_FP32_LAZY) {
    batch_points_kernel<true><<<g.points, kPointThreads, points_smem(c, true), s>>>(c, b);
    const int lp = std::min(c.log_pts, kLogPicks);
    const uint64_t warps = c.K * ((((c.child_stride + 31) >> 5) + (1u << lp) - 1) >> lp);
    const int grid = (int)std::min<uint64_t>((warps + 3) / 4, (uint64_t)g.picks);
    batch_picks_kernel<<<grid, kPointThreads, picks_smem(c), s>>>(c, b);
  } else {
    batch_points_kernel<false><<<g.points, kPointThreads, points_smem(c, false), s>>>(c, b);
  }
  return cudaGetLastError();
}

cudaError_t set_batch_tile_attributes(int max_smem)
{
  cudaError_t e = allow_dynamic_smem(batch_constraints_kernel<0, true>, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(batch_constraints_kernel<1, false>, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(batch_siblings_kernel, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(batch_lazy_kernel, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(batch_points_kernel<true>, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(batch_points_kernel<false>, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(batch_picks_kernel, max_smem);
  return e;
}

}  // namespace cmn
