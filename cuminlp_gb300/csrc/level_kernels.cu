// level_kernels.cu -- programs with shared slots over few boxes: a tile of 32
// boxes per block, lane = box, the program's runs in levels over the block's
// warps (Program::level_*), every slot of the tile in shared memory.
//
// What bounds it: with one lane per box a call of a few thousand boxes keeps
// one warp on a scheduler, and that warp walks the program at its latency (8
// cycles an instruction, 200 instructions a node of a model with divisions
// and roots).  Runs that do not read each other's results go to different
// warps here, with a barrier between levels.  Results do not change: every
// node is the same operation on the same operands.  3,001 host boxes of a
// model of 17 variables (204 instructions, 43 of them on the longest warp,
// 20 levels), copies included: 217 -> 105 us.
#include <cstdint>

#include "child_core.cuh"
#include "launch.hpp"

namespace cmn {

namespace {

size_t level_smem(const EvalArgs& a, bool fp32)
{
  const size_t t = fp32 ? 4 : 8, ms = a.pinfo != nullptr ? (size_t)a.max_slots : 0;
  return 32 * (2 * t * ((size_t)a.level.slots + ms) + 4 * ms);
}

}  // namespace

// kMode 0 of eval_children: boxes, or the regions of a role's box.
template <typename T>
__global__ void __launch_bounds__(kLevelWarps * 32) level_eval_kernel(const EvalArgs a)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned infeasible_s, excluded_s;
  __shared__ T obj_lo[32], obj_hi[32];
  T* base = reinterpret_cast<T*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ms = a.pinfo != nullptr ? a.max_slots : 0;
  Tile<T> t;
  t.lo = nullptr;
  t.hi = nullptr;
  t.slo = base;
  t.shi = base + (size_t)a.level.slots * 32;
  t.stride = 32;
  t.tid = lane;
  T* olo = base + (size_t)2 * a.level.slots * 32 + lane;
  T* ohi = olo + (size_t)ms * 32;
  int32_t* ovid = reinterpret_cast<int32_t*>(base + (size_t)2 * (a.level.slots + ms) * 32) + lane;
  const Instr* prog = sizeof(T) == 8 ? a.level.prog64 : a.level.prog32;
  const uint64_t total = a.n_children, tiles = (total + 31) >> 5;
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint64_t at = (tile << 5) + lane;
    const bool live = at < total;
    const uint64_t g = live ? at : total - 1;  // lanes past the end shadow the last box
    uint64_t k, r;
    child_of(a.log2C, g, k, r);
    if (threadIdx.x == 0) infeasible_s = excluded_s = 0;
    if (threadIdx.x < 32) obj_lo[lane] = obj_hi[lane] = Arith<T>::nan();
    bool dup;
    // every warp fills the tile's split columns with the same values
    const ChildVars<T, double> cv = child_vars<T, double>(a, a.plo, a.phi, k, r, olo, ohi, ovid, 32, dup);
    __syncthreads();
    Verdict<T> v = verdict_init<T>();
    for (int l = 0; l < a.level.levels; ++l) {
      const int j0 = __ldg(a.level.off + l * kLevelWarps + wid), j1 = __ldg(a.level.off + l * kLevelWarps + wid + 1);
      for (int j = j0; j < j1; ++j)
        interval_range<T>(prog, __ldg(a.level.run + 2 * j), __ldg(a.level.run + 2 * j + 1), cv, t, v);
      __syncthreads();
    }
    if (!v.feasible) atomicOr(&infeasible_s, 1u << lane);
    if (v.excluded) atomicOr(&excluded_s, 1u << lane);
    if (v.has_obj) {
      obj_lo[lane] = v.obj.lo;
      obj_hi[lane] = v.obj.hi;
    }
    __syncthreads();
    if (wid == 0 && live) {
      v.feasible = !((infeasible_s >> lane) & 1u);
      v.excluded = (excluded_s >> lane) & 1u;
      v.obj.lo = obj_lo[lane];
      v.obj.hi = obj_hi[lane];
      write_verdict<T, 0>(a, g, k, v, 0.0);
    }
    __syncthreads();  // the tile is restaged next
  }
}

// Up to four tiles an SM: beyond that every scheduler has warps of its own
// boxes, and the barriers and the slots' shared memory only cost.  Host boxes
// of 5 / 17 / 64 variables, copies included, levels against one lane per box:
// 19,456 boxes 108 / 189 / 613 against 122 / 252 / 756 us; at 30,000 one lane
// per box takes 129 / 280 / 832 and the levels, by their slope, as much.
bool level_fits(const EvalArgs& a, bool fp32)
{
  return a.level.levels > 0 && a.n_children_dev == nullptr && a.n_children > 0 && a.n_children <= (uint64_t)sm_count() * 4 * 32 &&
         level_smem(a, fp32) + 1024 <= (size_t)max_dynamic_smem();
}

cudaError_t launch_level(const EvalArgs& a, bool fp32, cudaStream_t s)
{
  const size_t smem = level_smem(a, fp32);
  const unsigned grid = (unsigned)((a.n_children + 31) >> 5);
  if (fp32) level_eval_kernel<float><<<grid, kLevelWarps * 32, smem, s>>>(a);
  else level_eval_kernel<double><<<grid, kLevelWarps * 32, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t set_level_kernel_attributes(int max_smem)
{
  cudaError_t e = allow_dynamic_smem(level_eval_kernel<double>, max_smem);
  return e == cudaSuccess ? allow_dynamic_smem(level_eval_kernel<float>, max_smem) : e;
}

}  // namespace cmn
