// child_core.cuh -- device code shared by the evaluators of children: which
// parent and region a child is, its variables, where its verdict goes, and
// the candidate reduction of the samplers.
#pragma once

#include <cfloat>
#include <cstdint>

#include "eval_core.cuh"
#include "kernels.cuh"
#include "stamps.cuh"

namespace cmn {

__device__ __forceinline__ void child_of(int log2C, uint64_t g, uint64_t& k, uint64_t& r)
{
  if (log2C < 0) {
    k = 0;
    r = g;
  } else {
    k = g >> log2C;
    r = g & ((1ULL << log2C) - 1ULL);
  }
}

// The variable source of child (k, r): the parent's planes `plo`/`phi`
// (FP64, or FP32 rounded outward) plus the child's split variables, decoded
// from the parent's FP64 bounds into this thread's columns olo/ohi/ovid.
// `dup` is set when a slot digit is at or past its domain size
// (region::is_duplicate_child).
template <typename T, typename S>
__device__ __forceinline__ ChildVars<T, S> child_vars(const EvalArgs& a, const S* plo, const S* phi, uint64_t k,
                                                      uint64_t r, T* olo, T* ohi, int32_t* ovid, int stride,
                                                      bool& dup)
{
  ChildVars<T, S> cv;
  cv.plo = plo + k;
  cv.phi = phi + k;
  cv.pstride = a.pstride;
  cv.mask = 0;
  cv.olo = olo;
  cv.ohi = ohi;
  cv.ovid = ovid;
  cv.count = 0;
  cv.stride = stride;
  dup = false;
  if (a.pinfo != nullptr) {
    const uint32_t count = a.pinfo[k].count;
    const SlotPlan* sp = a.slots + k * (uint64_t)a.max_slots;
    for (uint32_t j = 0; j < count; ++j) {
      const SlotPlan s = sp[j];
      const uint64_t part = slot_part(r, s);
      if (part >= s.dom) dup = true;
      double lo, hi;
      slot_bounds(s, a.plo[(uint64_t)s.vid * a.pstride + k], a.phi[(uint64_t)s.vid * a.pstride + k], part, lo, hi);
      olo[j * stride] = Widen<T, double>::lo(lo);
      ohi[j * stride] = Widen<T, double>::hi(hi);
      ovid[j * stride] = (int32_t)s.vid;
      cv.mask |= 1ULL << (s.vid & 63);
    }
    cv.count = (int)count;
  }
  return cv;
}

// Writes the verdict of child g of parent k (kModes as in eval_children).
template <typename T, int kMode>
__device__ __forceinline__ void write_verdict(const EvalArgs& a, uint64_t g, uint64_t k, const Verdict<T>& v,
                                              double gub)
{
  double lb = (double)v.obj.lo;
  if (kMode == 5 && a.parent_lb == nullptr) {
    // the solver's lazy form: the parent's FP64 verdict runs beside this
    // pass, and lazy_fold_kernel folds it in and settles every state but
    // these two
    a.out_lb[g] = lb;
    a.out_flag[g] = v.excluded ? kChildInfeasible : kChildScreened;
    return;
  }
  if (kMode == 5) {
    // the parent's certified bound holds for every child box inside it
    const double plb = a.parent_lb[k];
    lb = plb > lb ? plb : lb;
    a.out_lb[g] = lb;
    // a survivor whose bound lies within the band below the incumbent goes
    // to the FP64 pass, which may prune it; below the band FP64 could not
    a.out_flag[g] = v.excluded  ? kChildInfeasible
                    : lb > gub  ? kChildDominated
                    : lb >= certify_floor(gub) ? kChildScreened
                                               : kChildEligible;
    return;
  }
  if (kMode == 3 && a.parent_lb != nullptr) {  // lazy form's certify pass
    const double plb = a.parent_lb[k];
    lb = plb > lb ? plb : lb;
  }
  if (kMode == 0) {
    a.out_lb[g] = lb;
    if (a.out_ub) a.out_ub[g] = (double)v.obj.hi;
    // FP64: the reference predicate; FP32: not proven violated
    a.out_flag[g] = (uint8_t)(sizeof(T) == 8 ? v.feasible : !v.excluded);
  } else if (kMode == 2) {
    a.out_lb[g] = lb;
    a.out_flag[g] = v.excluded ? kChildInfeasible : (lb > gub ? kChildDominated : kChildScreened);
  } else {
    a.out_lb[g] = lb;
    a.out_flag[g] = !v.feasible ? kChildInfeasible : (lb > gub ? kChildDominated : kChildEligible);
  }
}

// Aggregate bounder (backend/aggregate/kernels.cuh:32-47 mask and the
// replay's per-child Min/Max, replay.cuh:497-556), fused: region r belongs
// to child r / agg_m; infeasible regions count as lb = +inf, ub = -inf.
// Minimum and maximum follow the total order of lb_key.  A warp whose
// active lanes share one child combines them before one pair of atomics.
// Every lane of the warp calls this.
__device__ __forceinline__ void aggregate_fold(const EvalArgs& a, bool active, uint64_t r, const Verdict<double>& v)
{
  const unsigned c = active ? (unsigned)(r / a.agg_m) : 0xffffffffu;
  unsigned long long kmin = lb_key(active && v.feasible ? v.obj.lo : INFINITY);
  unsigned long long kmax = lb_key(active && v.feasible ? v.obj.hi : -INFINITY);
  const unsigned any = __ballot_sync(0xffffffffu, active);
  if (any == 0) return;
  const unsigned cmin = __reduce_min_sync(0xffffffffu, c);
  const unsigned cmax = __reduce_max_sync(0xffffffffu, active ? c : 0u);
  if (cmin == cmax) {
    for (int off = 16; off > 0; off >>= 1) {
      const unsigned long long a1 = __shfl_xor_sync(0xffffffffu, kmin, off);
      const unsigned long long b1 = __shfl_xor_sync(0xffffffffu, kmax, off);
      kmin = a1 < kmin ? a1 : kmin;
      kmax = b1 > kmax ? b1 : kmax;
    }
    if ((threadIdx.x & 31) == (unsigned)(__ffs(any) - 1)) {
      atomicMin(a.agg_keys + cmin, kmin);
      atomicMax(a.agg_keys + a.agg_k + cmin, kmax);
    }
  } else if (active) {
    atomicMin(a.agg_keys + c, kmin);
    atomicMax(a.agg_keys + a.agg_k + c, kmax);
  }
}

__device__ __forceinline__ void warp_min_cand(Cand& c)
{
  for (int off = 16; off > 0; off >>= 1) {
    Cand o;
    o.value = __shfl_down_sync(0xffffffffu, c.value, off);
    o.k = __shfl_down_sync(0xffffffffu, c.k, off);
    o.e = __shfl_down_sync(0xffffffffu, c.e, off);
    o.pad = 0;
    if (cand_less(o, c)) c = o;
  }
}

// Block-wide min of one Cand per thread; result valid in thread 0.
__device__ __forceinline__ Cand block_min_cand(Cand c)
{
  __shared__ Cand warp_best[32];
  warp_min_cand(c);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) warp_best[wid] = c;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  if (wid == 0) {
    Cand x = lane < nw ? warp_best[lane] : Cand{INFINITY, 0xffffffffu, 0, ~0ULL};
    warp_min_cand(x);
    c = x;
  }
  __syncthreads();
  return c;
}

}  // namespace cmn
