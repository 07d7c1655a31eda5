// chain32_kernels.cu -- the FP32 passes over programs of sum chains for one
// instance (chain32_tiles.cuh).
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "chain32_tiles.cuh"
#include "launch.hpp"

namespace cmn {

// kMode 0: boxes -> out_lb, out_ub, out_flag = not proven violated; 2: the
// screen of the solver's children -> out_lb, out_flag = ChildState.
template <int kMode>
__global__ void __launch_bounds__(kWarps32 * 32, 4) chain32_eval_kernel(const EvalArgs a)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned excluded_s, bad_s;
  __shared__ int next_s;
  __shared__ float lo_s[32], hi_s[32];
  float2* x = reinterpret_cast<float2*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int n = a.n_vars;
  if (a.done != nullptr && *a.done) return;
  const uint64_t total = a.n_children_dev ? *a.n_children_dev : a.n_children;
  const double gub = a.gub ? *a.gub : DBL_MAX;
  const bool pass_through = kMode == 2 && a.use_screen != nullptr && *a.use_screen == 0;
  const bool want_hi = kMode == 0 && a.out_ub != nullptr;
  const uint64_t tiles = (total + 31) >> 5;
  if (wid == 0) x[n * 32 + lane] = make_float2(1.0f, 1.0f);  // linear terms
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint64_t at = (tile << 5) + lane;
    bool live = at < total;
    const uint64_t g = live ? at : total - 1;
    uint64_t k, r;
    child_of(a.log2C, g, k, r);
    uint32_t count = 0;
    const SlotPlan* sp = nullptr;
    if (kMode == 2) {
      const ParentInfo pi = a.pinfo[k];
      count = pi.count;
      sp = a.slots + k * (uint64_t)a.max_slots;
      if (pi.fathom || r >= pi.nreg) {
        if (live && wid == 0) a.out_flag[g] = kChildNone;
        live = false;
      }
      bool dup = false;
      for (uint32_t j = 0; j < count; ++j) dup = dup || slot_part(r, sp[j]) >= sp[j].dom;
      if (live && (dup || pass_through)) {
        if (wid == 0) a.out_flag[g] = dup ? kChildDuplicate : kChildScreened;
        live = false;
      }
    }
    const unsigned alive = __ballot_sync(0xffffffffu, live);  // the same in every warp
    if (alive == 0u) continue;
    bool bad = false;
    for (int v = wid; v < n; v += W) {
      const uint64_t o = (uint64_t)v * a.pstride + k;
      float2 p;
      if (a.plo32 != nullptr) p = make_float2(__ldg(a.plo32 + o), __ldg(a.phi32 + o));
      else p = make_float2(__double2float_rd(__ldg(a.plo + o)), __double2float_ru(__ldg(a.phi + o)));
      x[v * 32 + lane] = p;
      bad = bad || out_of_range(p);
    }
    if (threadIdx.x == 0) {
      excluded_s = 0;
      bad_s = 0;
      next_s = 0;
    }
    __syncthreads();
    for (uint32_t j = wid; j < count; j += W) {
      const SlotPlan s = sp[j];
      bool leads = true;  // a variable of two slots takes the first one's part
      for (uint32_t q = 0; q < j; ++q) leads = leads && sp[q].vid != s.vid;
      if (!leads) continue;
      double lo, hi;
      slot_bounds(s, a.plo[(uint64_t)s.vid * a.pstride + k], a.phi[(uint64_t)s.vid * a.pstride + k], slot_part(r, s), lo, hi);
      const float2 p = make_float2(__double2float_rd(lo), __double2float_ru(hi));
      x[s.vid * 32 + lane] = p;
      bad = bad || out_of_range(p);
    }
    if (bad) atomicOr(&bad_s, 1u << lane);
    __syncthreads();
    // the chains, the objective's upper bound beside its lower one
    for (;;) {
      int q = 0;
      if (lane == 0) q = atomicAdd(&next_s, 1);
      q = __shfl_sync(0xffffffffu, q, 0) - (want_hi ? 1 : 0);
      if (q >= a.chain.n_seg) break;
      const ChainSeg& s = a.chain.seg[q < 0 ? 0 : q];
      if (q < 0) {
        hi_s[lane] = chain32<true>(a.chain.term32, s.t32, s.t32_end, x + lane);
        continue;
      }
      const float lo = chain32<false>(a.chain.term32, s.t32, s.t32_end, x + lane);
      if (s.kind == kChainObjective) {
        lo_s[lane] = lo;
      } else {
        // lo > rhs, exactly: rhs_dn is the largest float not above rhs
        const unsigned no = __ballot_sync(0xffffffffu, lo > s.rhs_dn);
        if (lane == 0 && no) atomicOr(&excluded_s, no);
      }
    }
    __syncthreads();
    if (wid == 0 && live) {
      Verdict<float> v = verdict_init<float>();
      v.excluded = (excluded_s >> lane) & 1u;
      v.obj.lo = lo_s[lane];
      if (want_hi) v.obj.hi = hi_s[lane];
      if ((bad_s >> lane) & 1u) v = box_general(a.prog, a.prog_len, TileVars{x + lane});
      write_verdict<float, kMode>(a, g, k, v, gub);
    }
    __syncthreads();  // the tile is restaged next
  }
}

__global__ void __launch_bounds__(kLazyThreads, 2) lazy_children_kernel(const EvalArgs a, const LazyShape h)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LazyShared sh;
  if (a.done != nullptr && *a.done) return;
  const uint64_t E = *a.n_parents_dev, tiles = (E + 31) >> 5;
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) lazy_tile(a, h, smem_raw, sh, tile, E);
  if (threadIdx.x == 0) stamp_last(a.t_last, blockIdx.x < tiles);
}

// ---- launchers ----
static size_t eval32_smem(int n) { return (size_t)(n + 1) * 32 * 8; }

bool chain32_fits(const EvalArgs& a, int mode)
{
  return a.chain.term32 != nullptr && (mode == 0 ? a.pinfo == nullptr : mode == 2) &&
         eval32_smem(a.n_vars) + 1024 <= (size_t)max_dynamic_smem();
}

// Whether the tiles beat the interpreter over boxes (the screen always takes
// them).  Up to one wave they do.  Beyond, a tile waits for its variables with
// the few warps that its shared memory leaves an SM, so the terms have to
// outweigh that (a product counts 2.4: the interpreter takes that much longer
// for it): a linear objective, n = 64, 12 warps, 65,536 boxes 40 us by the
// interpreter and 67 in tiles; n = 150, 301 terms, 5 warps, 200,000 boxes 985
// and 1,231; n = 300 with two linear constraints, 6 warps, 20,000 boxes 201 and
// 283; n = 100, 201 terms, 8 warps, 200,000 boxes 608 and 565.  Programs of
// less than 12 instructions take launch time either way (11 and 12 us) up to
// some 10^5 boxes (n = 2, 6 instructions, 524,288 boxes 26 and 22).
bool chain32_pays(const EvalArgs& a, int mode)
{
  if (mode != 0) return true;
  const int64_t len = a.prog_len, n = a.n_vars, boxes = (int64_t)a.max_boxes;
  if (len < 12) return len >= 6 && boxes >= 131072 && 5 * len >= 6 * n;
  const int64_t tiles = std::min<int64_t>(32, max_dynamic_smem() / (int64_t)(eval32_smem(a.n_vars) + 1024));
  return boxes <= 32 * tiles * sm_count() || (10 * len + 14ll * a.chain.products) * tiles * a.chain.warps32 >= 250 * n;
}

template <int kMode>
static cudaError_t launch_chain32_t(const EvalArgs& a, cudaStream_t s)
{
  const size_t smem = eval32_smem(a.n_vars);
  const int threads = 32 * a.chain.warps32;
  const uint64_t grid = resident_blocks((a.max_boxes + 31) >> 5, chain32_eval_kernel<kMode>, threads, smem);
  chain32_eval_kernel<kMode><<<(unsigned)grid, threads, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_chain32(const EvalArgs& a, int mode, cudaStream_t s)
{
  return mode == 0 ? launch_chain32_t<0>(a, s) : launch_chain32_t<2>(a, s);
}

// As many chains per round as keep two blocks on an SM, none fewer than four;
// {0, 0} when the parents' tables do not fit.
static LazyShape lazy_shape(int n, int ms, int log2C, int chains)
{
  if (ms > kLazySlots || log2C > kLazySlots) return LazyShape{0, 0};
  const size_t room = (size_t)max_dynamic_smem() - 2048;
  const int children = 1 << log2C;
  LazyShape h = {chains, (1 << log2C) + 1};
  while (h.chains > 4 && lazy_smem(n, ms, h, children) > room / 2) h.chains = (h.chains + 1) / 2;
  if (lazy_smem(n, ms, h, children) > room) h.chains = 0;
  return h;
}

bool lazy_children_fits(const ChainTab& t, int n, int ms, int log2C)
{
  return t.term32 != nullptr && lazy_shape(n, ms, log2C, t.n_seg).chains > 0;
}

cudaError_t launch_lazy_children(const EvalArgs& a, uint64_t max_parents, cudaStream_t s)
{
  const LazyShape h = lazy_shape(a.n_vars, a.max_slots, a.log2C, a.chain.n_seg);
  const size_t smem = lazy_smem(a.n_vars, a.max_slots, h, 1 << a.log2C);
  const uint64_t grid = resident_blocks((max_parents + 31) >> 5, lazy_children_kernel, kLazyThreads, smem);
  lazy_children_kernel<<<(unsigned)grid, kLazyThreads, smem, s>>>(a, h);
  return cudaGetLastError();
}

cudaError_t set_chain32_kernel_attributes(int max_smem)
{
  cudaError_t e = allow_dynamic_smem(chain32_eval_kernel<0>, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(chain32_eval_kernel<2>, max_smem);
  if (e == cudaSuccess) e = allow_dynamic_smem(lazy_children_kernel, max_smem);
  return e;
}

}  // namespace cmn
