// chain32_tiles.cuh -- the FP32 passes over programs of sum chains: the
// outward-rounded enclosures of boxes and children (the screen), and the
// lazy form's child bounds from incremental chain sums.  A tile of 32 boxes
// or parents per block, a warp per chain, lane = box, the boxes' bounds in
// shared memory.
//
// What bounds them: FP32 issue and shared-memory loads (two of 8 bytes per
// term and box).  A constraint carries its lower bound alone and the
// objective the bounds that are read, with the roundings the interpreter
// gives them.
#pragma once

#include <cfloat>
#include <cstdint>

#include "chain_core.cuh"
#include "child_core.cuh"

namespace cmn {

constexpr int kWarps32 = 8;     // warps of an evaluation tile at most
constexpr int kLazyThreads = 512;
constexpr int kLazySlots = 6;   // most slots per parent of the lazy pass

// Whether a bound is outside the range of the fast term arithmetic, or the
// pair is no interval: within it no product overflows or underflows, so the
// extreme of the four directed corner products is the tightest bound, as the
// interpreter's sign classes give it.
__device__ __forceinline__ bool out_of_range(float2 p)
{
  const uint32_t a = __float_as_uint(p.x) & 0x7fffffffu, b = __float_as_uint(p.y) & 0x7fffffffu;
  return p.x > p.y || (a != 0u && (a - (87u << 23)) >= (80u << 23)) ||  // [2^-40, 2^40)
         (b != 0u && (b - (87u << 23)) >= (80u << 23));
}

// The lower (kUp: upper) end of one term over x_a in A and x_b in B.
template <bool kUp>
__device__ __forceinline__ float term_end(const uint4 t, float2 A, float2 B)
{
  const uint32_t flip = t.y & kT32Neg;
  const float cl = __uint_as_float(t.z), ch = __uint_as_float(t.w);
  float q;
  if (t.y & kT32Sqr) {
    const bool neg = flip != 0u;
    if (neg != kUp) {
      const float m = fmaxf(-A.x, A.y);
      q = __fmul_ru(m, m);
    } else {
      const float d = fmaxf(fmaxf(A.x, -A.y), 0.0f);
      q = __fmul_rd(d, d);
    }
    q = __uint_as_float(__float_as_uint(q) ^ flip);
  } else {
    const float ax = __uint_as_float(__float_as_uint(A.x) ^ flip), ay = __uint_as_float(__float_as_uint(A.y) ^ flip);
    q = kUp ? max4(__fmul_ru(ax, B.x), __fmul_ru(ax, B.y), __fmul_ru(ay, B.x), __fmul_ru(ay, B.y))
            : min4(__fmul_rd(ax, B.x), __fmul_rd(ax, B.y), __fmul_rd(ay, B.x), __fmul_rd(ay, B.y));
  }
  return kUp ? fmaxf(__fmul_ru(cl, q), __fmul_ru(ch, q)) : fminf(__fmul_rd(cl, q), __fmul_rd(ch, q));
}

// acc + the term, rounded towards the bound.  A zero product counts as +0
// (a zero factor gives +0), whatever its corners' signs.
template <bool kUp>
__device__ __forceinline__ float term_add(float acc, const uint4 t, float2 A, float2 B)
{
  if ((t.y & (kT32Sub | kT32Raw | kT32Const)) == 0u) {
    const float e = term_end<kUp>(t, A, B) + 0.0f;
    return kUp ? __fadd_ru(acc, e) : __fadd_rd(acc, e);
  }
  if (t.y & kT32Const) return kUp ? __fadd_ru(acc, __uint_as_float(t.w)) : __fadd_rd(acc, __uint_as_float(t.z));
  float e = term_end<kUp>(t, A, B);
  if (t.y & kT32Sub) {
    e = -e;
    if (!(t.y & kT32Raw)) e += 0.0f;
    return kUp ? __fsub_ru(acc, e) : __fsub_rd(acc, e);
  }
  return kUp ? __fadd_ru(acc, e) : __fadd_rd(acc, e);
}

// One bound of the chain over the box at x (a float2 per variable, 32 apart).
template <bool kUp>
__device__ __forceinline__ float chain32(const ChainTerm32* __restrict__ term, int t0, int t1,
                                         const float2* __restrict__ x)
{
  const uint4* __restrict__ w = reinterpret_cast<const uint4*>(term);
  float acc = 0.0f;
  int q = t0;
  // four plain terms at a time: their loads and products before the first add
  for (; q + 4 <= t1; q += 4) {
    uint4 t[4];
    uint32_t special = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      t[u] = __ldg(w + q + u);
      special |= t[u].y;
    }
    if ((special & (kT32Sub | kT32Raw | kT32Const)) == 0u) {
      float e[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) e[u] = term_end<kUp>(t[u], x[(t[u].x & 0xffffu) * 32], x[(t[u].x >> 16) * 32]) + 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u) acc = kUp ? __fadd_ru(acc, e[u]) : __fadd_rd(acc, e[u]);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) acc = term_add<kUp>(acc, t[u], x[(t[u].x & 0xffffu) * 32], x[(t[u].x >> 16) * 32]);
    }
  }
  for (; q < t1; ++q) {
    const uint4 t = __ldg(w + q);
    acc = term_add<kUp>(acc, t, x[(t.x & 0xffffu) * 32], x[(t.x >> 16) * 32]);
  }
  return acc;
}

// A tile's box out of range: the interpreter's verdict.
template <typename V>
static __device__ __noinline__ Verdict<float> box_general(const Instr* prog, int len, const V& vars)
{
  const Tile<float> t = {};
  return run_interval<float, V>(prog, len, vars, t);
}

// The box in a tile, for the interpreter.
struct TileVars {
  const float2* x;
  __device__ __forceinline__ Iv<float> var(int v) const
  {
    const float2 p = x[v * 32];
    return {p.x, p.y};
  }
};


// ---- the lazy form's child bounds ----
// Per tile of 32 parents: (1) the common sum of every chain, its terms that
// read no variable the parent splits; (2) the part sums of every chain and
// slot part, the terms that read that slot's variable over the part and no
// variable of an earlier slot; (3) every child adds, per chain, its slots'
// part sums to the common one.  All three stay in shared memory: through
// global memory the part sums alone were 128 bytes a child.
//
// inc_common_kernel, inc_parts_kernel and eval_children_inc_kernel give the
// same sums for programs with other readers or more slots.  n = 64 MIQCQP,
// the 13 iterations of a solve with 2^16 parents x 2^4 children: the three
// took 44.1 ms, this pass 11.7.
struct LazyShape {
  int chains;  // chains per round of the three steps
  int parts;   // parts per parent at most (2^B), and one to spread the banks
};

inline __host__ __device__ size_t lazy_smem(int n, int ms, LazyShape h, int children)
{
  return (size_t)(n + 1) * 32 * 8 * 2 + (size_t)h.parts * 32 * 8 + (size_t)ms * 32 * 4 +
         (size_t)h.chains * 32 * 4 * (1 + (size_t)h.parts) + (size_t)children * 32 * 5;
}

// A parent out of range: its sums by the interpreter's arithmetic.
struct ParentVars {
  const float2* x;
  int vid;  // -1: the parent's own bounds everywhere
  Iv<float> val;
  __device__ __forceinline__ Iv<float> var(int v) const
  {
    if (v == vid) return val;
    const float2 p = x[v * 32];
    return {p.x, p.y};
  }
};

// The terms [pc0, pc1) of one chain that a sum takes: the common one
// (`slot` < 0) leaves out every split variable, a part sum takes the terms of
// its slot's variable and leaves out earlier slots'.
static __device__ __noinline__ float sum_general(const Instr* prog, int pc0, int pc1, const ParentVars& vars,
                                          const int32_t* svid, int count, int slot)
{
  Iv<float> acc = {0.0f, 0.0f};
  auto split_before = [&](int v, int j) {
    for (int q = 0; q < j; ++q)
      if (svid[q * 32] == v) return true;
    return false;
  };
  for (int pc = pc0; pc < pc1; ++pc) {
    const Instr cur = load_instr(prog, pc);
    const int code = cur.head & 7;
    const bool reads = code == kOpTerm || (cur.modes & 3) == kModeVar;
    if (slot < 0) {
      if (reads && (split_before(cur.a, count) || (code == kOpTerm && split_before(cur.b, count)))) continue;
    } else {
      if (!reads) continue;
      const bool at_a = cur.a == vars.vid, at_b = code == kOpTerm && cur.b == vars.vid;
      if (!at_a && !at_b) continue;
      const int other = at_a ? (code == kOpTerm ? (int)cur.b : (int)cur.a) : (int)cur.a;
      if (other != vars.vid && split_before(other, slot)) continue;
    }
    acc = chain_add<float, ParentVars>(acc, cur, vars);
  }
  return acc.lo;
}

struct LazyShared {
  unsigned bad;
  int next;
};

// One tile of 32 parents of the E; the whole block calls this for the same.
__device__ __forceinline__ void lazy_tile(const EvalArgs& a, const LazyShape& h, unsigned char* smem, LazyShared& sh,
                                          uint64_t tile, uint64_t E)
{
  const int n = a.n_vars, ms = a.max_slots;
  const int lane = threadIdx.x & 31, W = blockDim.x >> 5;
  const int C = 1 << a.log2C, NC = 32 * C;
  float2* x = reinterpret_cast<float2*>(smem);        // the parents' bounds
  float2* xc = x + (size_t)(n + 1) * 32;                  // split variables zero: they add nothing
  float2* xp = xc + (size_t)(n + 1) * 32;                 // [parts][32] split variable over each part
  int32_t* svid = reinterpret_cast<int32_t*>(xp + (size_t)h.parts * 32);  // [ms][32]
  float* common = reinterpret_cast<float*>(svid + (size_t)ms * 32);       // [chain][32]
  float* part = common + (size_t)h.chains * 32;                           // [chain][32][parts]
  float* child_lb = part + (size_t)h.chains * 32 * h.parts;               // [32 * C]
  uint8_t* child_ex = reinterpret_cast<uint8_t*>(child_lb + NC);
  const int wid = threadIdx.x >> 5;
  const int S = a.chain.n_seg;
  const double gub = a.gub ? *a.gub : DBL_MAX;
  const uint4* __restrict__ var32 = reinterpret_cast<const uint4*>(a.chain.var32);
  if (wid == 0) x[n * 32 + lane] = xc[n * 32 + lane] = make_float2(1.0f, 1.0f);  // linear terms
  const uint64_t kat = (tile << 5) + lane;
  const uint64_t k = kat < E ? kat : E - 1;  // lanes past the end shadow the last parent
  const ParentInfo pi = a.pinfo[k];
  const SlotPlan* sp = a.slots + k * (uint64_t)ms;
  const int count = (int)pi.count;
  bool bad = false;
  for (int v = wid; v < n; v += W) {
    const uint64_t o = (uint64_t)v * a.pstride + k;
    const float2 p = make_float2(__ldg(a.plo32 + o), __ldg(a.phi32 + o));
    x[v * 32 + lane] = p;
    xc[v * 32 + lane] = p;
    bad = bad || out_of_range(p);
  }
  if (threadIdx.x == 0) sh.bad = 0;
  __syncthreads();
  // slots: the split variables, and each over its parts
  uint64_t split = 0;
  int ubase = 0;
  for (int j = 0; j < count; ++j) {
    const SlotPlan s = sp[j];
    split |= 1ULL << (s.vid & 63);
    if (wid == 0) {
      svid[j * 32 + lane] = (int32_t)s.vid;
      xc[s.vid * 32 + lane] = make_float2(0.0f, 0.0f);
    }
    for (int p = wid; p < (int)s.width && ubase + p < h.parts; p += W) {
      double lo, hi;
      slot_bounds(s, a.plo[(uint64_t)s.vid * a.pstride + k], a.phi[(uint64_t)s.vid * a.pstride + k], (uint64_t)p, lo, hi);
      const float2 q = make_float2(__double2float_rd(lo), __double2float_ru(hi));
      xp[(ubase + p) * 32 + lane] = q;
      bad = bad || out_of_range(q);
    }
    ubase += (int)s.width;
  }
  if (bad) atomicOr(&sh.bad, 1u << lane);
  for (int c = threadIdx.x; c < NC; c += blockDim.x) child_ex[c] = 0;
  for (int s0 = 0; s0 < S; s0 += h.chains) {
    const int sn = S - s0 < h.chains ? S - s0 : h.chains;
    if (threadIdx.x == 0) sh.next = 0;
    __syncthreads();
    const bool general = (sh.bad >> lane) & 1u;
    for (;;) {
      int it = 0;
      if (lane == 0) it = atomicAdd(&sh.next, 1);
      it = __shfl_sync(0xffffffffu, it, 0);
      if (it >= sn * (1 + ms)) break;
      if (it < sn) {  // (1) common sums
        const ChainSeg& s = a.chain.seg[s0 + it];
        float acc = chain32<false>(a.chain.term32, s.t32, s.t32_end, xc + lane);
        if (general) acc = sum_general(a.prog, s.pc0, s.pc1, ParentVars{x + lane, -1, {0.0f, 0.0f}}, svid + lane, count, -1);
        common[it * 32 + lane] = acc;
        continue;
      }
      // (2) part sums: slot j of chain c, two parts at a time
      const int c = (it - sn) / ms, j = (it - sn) - c * ms;
      if (j >= count) continue;
      const int v = svid[j * 32 + lane];
      uint64_t earlier = 0;
      bool repeated = false;
      int ub = 0;
      for (int q = 0; q < j; ++q) {
        const int w = svid[q * 32 + lane];
        earlier |= 1ULL << (w & 63);
        repeated = repeated || w == v;
        ub += (int)sp[q].width;
      }
      const int width = (int)sp[j].width;
      const ChainSeg& s = a.chain.seg[s0 + c];
      const int q0 = __ldg(a.chain.var_off + (int64_t)v * S + s0 + c), q1 = __ldg(a.chain.var_off + (int64_t)v * S + s0 + c + 1);
      float* out = part + ((size_t)c * 32 + lane) * h.parts + ub;
      for (int p = 0; p < width; p += 2) {
        const float2 v0 = xp[(ub + p) * 32 + lane], v1 = xp[(ub + (p + 1 < width ? p + 1 : p)) * 32 + lane];
        float acc0 = 0.0f, acc1 = 0.0f;
        if (general && !repeated) {
          acc0 = sum_general(a.prog, s.pc0, s.pc1, ParentVars{x + lane, v, {v0.x, v0.y}}, svid + lane, count, j);
          acc1 = sum_general(a.prog, s.pc0, s.pc1, ParentVars{x + lane, v, {v1.x, v1.y}}, svid + lane, count, j);
        } else if (!repeated) {
          for (int q = q0; q < q1; ++q) {
            const uint4 t = __ldg(var32 + q);
            const int other = (int)(t.x >> 16);
            bool skip = false;
            if (other != v && ((earlier >> (other & 63)) & 1ULL))
              for (int e = 0; e < j; ++e) skip = skip || svid[e * 32 + lane] == other;
            if (skip) continue;  // that slot's part sum has it
            const float2 xo = x[other * 32 + lane];
            acc0 = term_add<false>(acc0, t, v0, other == v ? v0 : xo);
            acc1 = term_add<false>(acc1, t, v1, other == v ? v1 : xo);
          }
        }
        out[p] = acc0;
        if (p + 1 < width) out[p + 1] = acc1;
      }
    }
    __syncthreads();
    // (3) the children, lane = child
    for (int c = threadIdx.x; c < NC; c += blockDim.x) {
      const int kl = c >> a.log2C;
      const uint64_t ck = (tile << 5) + kl, r = (uint64_t)(c & (C - 1));
      if (ck >= E) break;  // the tile's parents end here
      const ParentInfo cp = a.pinfo[ck];
      if (cp.fathom || r >= cp.nreg) {
        if (s0 == 0) a.out_flag[(ck << a.log2C) + r] = kChildNone;
        continue;
      }
      const SlotPlan* cs = a.slots + ck * (uint64_t)ms;
      int u[kLazySlots];
      bool dup = false;
      int ub = 0;
#pragma unroll
      for (int j = 0; j < kLazySlots; ++j) {
        u[j] = -1;
        if (j < (int)cp.count) {
          const uint64_t p = slot_part(r, cs[j]);
          dup = dup || p >= cs[j].dom;
          u[j] = ub + (int)p;
          ub += (int)cs[j].width;
        }
      }
      if (dup) {
        if (s0 == 0) a.out_flag[(ck << a.log2C) + r] = kChildDuplicate;
        continue;
      }
      bool ex = child_ex[c] != 0;
      for (int q = 0; q < sn; ++q) {
        float acc = common[q * 32 + kl];
        const float* ps = part + ((size_t)q * 32 + kl) * h.parts;
#pragma unroll
        for (int j = 0; j < kLazySlots; ++j)
          if (u[j] >= 0) acc = __fadd_rd(acc, ps[u[j]]);
        if (s0 + q == 0) child_lb[c] = acc;  // the objective's chain is the first
        else ex = ex || acc > a.chain.seg[s0 + q].rhs_dn;
      }
      child_ex[c] = ex ? 1 : 0;
      if (s0 + sn == S) {
        Verdict<float> v = verdict_init<float>();
        v.excluded = ex;
        v.obj.lo = child_lb[c];
        write_verdict<float, 5>(a, (ck << a.log2C) + r, ck, v, gub);
      }
    }
    __syncthreads();  // the sums are refilled next
  }
}

}  // namespace cmn
