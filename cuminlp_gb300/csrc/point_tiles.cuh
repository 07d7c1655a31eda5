// point_tiles.cuh -- points of programs that are sets of sum chains: the
// sampler (and exact points), and the lazy form's FP32 sample screen.
//
// A warp draws a tile of points into shared memory and tests the constraints
// one after the other.  Most points fail an early one, and a lane per point
// would leave the warp running for its last survivor: on the n = 64 MIQCQP
// the last of 32 points fell to the twentieth constraint on average, a point
// alone to the fifth.  So the lanes are dealt anew over the points still in,
// as many as fit on each.
#pragma once

#include <cfloat>
#include <cstdint>

#include "chain_core.cuh"
#include "child_core.cuh"

namespace cmn {

constexpr int kPointThreads = 128;
// Bytes of a warp's FP32 points: fewer points, of more lanes each, for many
// variables, so that a block of four warps keeps within about 36 KiB (32
// points up to 71 variables).
constexpr size_t kPointBytes = 9 * 1024;

inline int log_points(int n)
{
  int lp = 5;
  while (lp > 0 && ((size_t)n * 4) << lp > kPointBytes) --lp;
  return lp;
}

// an odd distance between a variable's points and the next one's: lanes that
// share a point then read different banks
__host__ __device__ __forceinline__ int point_stride(int log_pts) { return (1 << log_pts) | 1; }

__host__ __device__ __forceinline__ size_t point_bytes(int n, int log_pts)
{
  return ((size_t)n * 4 * point_stride(log_pts) + 7) & ~(size_t)7;
}

__device__ __forceinline__ double key_value(uint64_t k)  // lb_key's inverse
{
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffULL) : ~k));
}

// x * 2^-53 for x < 2^53, exactly, on the integer pipe (the conversion and
// the product issue at the FP64 rate).
__device__ __forceinline__ double unit53(uint64_t x)
{
  if (x == 0) return 0.0;
  const int lz = __clzll((long long)x);  // >= 11
  return __longlong_as_double((long long)(((uint64_t)(1033 - lz) << 52) | ((x << lz << 1) >> 12)));
}

// sample_value with the draw from unit53
__device__ __forceinline__ double draw(bool discrete, double lb, double ub, uint64_t vid, uint64_t i, uint64_t region,
                                       uint64_t salt)
{
  if (discrete) return sample_value(true, lb, ub, vid, i, region, salt);
  return __fma_rn(unit53(sample_hash(vid, i, region, salt) >> 11), __dsub_rn(ub, lb), lb);
}

// What a point is drawn from.
struct PointOf {
  uint64_t k, r, i, salt;
  const SlotPlan* sp;
  uint32_t count;
  bool fathom;
};

__device__ __forceinline__ double coordinate(const SampleArgs& a, const PointOf& p, int v)
{
  double lo = a.plo[(uint64_t)v * a.pstride + p.k], hi = a.phi[(uint64_t)v * a.pstride + p.k];
  for (uint32_t j = 0; j < p.count; ++j)
    if (p.sp[j].vid == (uint32_t)v) {
      slot_bounds(p.sp[j], lo, hi, slot_part(p.r, p.sp[j]), lo, hi);
      break;
    }
  return p.fathom ? lo : draw(a.var_kinds[v] != 0, lo, hi, (uint64_t)v, p.i, p.r, p.salt);
}

// The child g's place and whether its points are taken; false: none.
__device__ __forceinline__ bool point_child(const SampleArgs& a, uint64_t g, uint64_t salt_base, PointOf& p)
{
  child_of(a.log2C, g, p.k, p.r);
  p.fathom = a.exact != 0;
  p.count = 0;
  p.sp = nullptr;
  p.salt = a.salt_base_dev ? salt_base + p.k + 1 : a.salt;
  if (a.pinfo != nullptr) {
    const ParentInfo pi = a.pinfo[p.k];
    p.fathom = p.fathom || pi.fathom;
    p.count = pi.count;
    p.sp = a.slots + p.k * (uint64_t)a.max_slots;
    if (p.r >= pi.nreg) return false;
  }
  if (a.state != nullptr && !p.fathom) {
    const uint8_t st = a.state[g] & 0x7f;  // the batch marks certified children in the top bit
    return a.sample_all ? (st != kChildNone) : (st == kChildEligible);
  }
  return true;
}

// The lanes of a warp dealt over the points of `alive`: L = 2^lg lanes on
// each, this lane the `sub`-th of point `pt` (pt < 0: none).
struct Deal {
  int pt, sub, lg;
};

__device__ __forceinline__ Deal deal(unsigned alive, uint8_t* list)
{
  const int lane = threadIdx.x & 31, A = __popc(alive);
  if ((alive >> lane) & 1u) list[__popc(alive & ((1u << lane) - 1u))] = (uint8_t)lane;
  __syncwarp();
  Deal d;
  d.lg = 0;
  while ((A << (d.lg + 1)) <= 32) ++d.lg;
  const int at = lane >> d.lg;
  d.pt = at < A ? list[at] : -1;
  d.sub = lane & ((1 << d.lg) - 1);
  __syncwarp();
  return d;
}

// This lane's share of one chain at the point x (one cut coordinate per
// variable, `stride` apart) and of its terms' magnitudes.
__device__ __forceinline__ void filter_point(const ChainSeg& s, const ChainTerm* __restrict__ term,
                                             const float* __restrict__ x, uint32_t stride, int sub, int L, float& sum,
                                             float& mag)
{
  float acc[2] = {sub == 0 ? s.c0 : 0.0f, 0.0f}, m[2] = {sub == 0 ? fabsf(s.c0) : 0.0f, 0.0f};
  auto add = [&](int u, float t) {
    acc[u] += t;
    m[u] += fabsf(t);
  };
  filter_group(term, s.group[0], s.group[2], sub, L, [&](int u, uint32_t a, uint32_t b, float c) {
    add(u, c * (x[a * stride] * x[b * stride]));
  });
  filter_group(term, s.group[2], s.group[4], sub, L, [&](int u, uint32_t a, uint32_t, float c) {
    const float p = x[a * stride];
    add(u, c * (p * p));
  });
  filter_group(term, s.group[4], s.group[6], sub, L, [&](int u, uint32_t a, uint32_t, float c) { add(u, c * x[a * stride]); });
  sum = acc[0] + acc[1];
  mag = m[0] + m[1];
}

// One term of the FP64 point program: [c *] (x_a [* x_b]), each operation
// rounded to nearest, negated when it is subtracted.
__device__ __forceinline__ double point_term(const Instr& cur, const double* __restrict__ x)
{
  const int sub = cur.head >> 3, pk = sub & kTermPMask;
  double p = x[cur.a];
  if (pk == kTermProd) p = __dmul_rn(p, x[cur.b]);
  else if (pk == kTermSqr) p = __dmul_rn(p, p);
  if (sub & kTermHasC) p = __dmul_rn(cur.c, p);
  return (sub & kTermSub) && !(sub & kTermInit) ? -p : p;
}

// The chain's FP64 value at the point x by a whole warp: 32 terms at once,
// then every lane adds them in order.
__device__ __forceinline__ double point_chain_warp(const Instr* __restrict__ prog, int pc0, int pc1,
                                                   const double* __restrict__ x)
{
  const int lane = threadIdx.x & 31;
  const Instr first = load_instr(prog, pc0);
  double acc = (first.head & 7) == kOpLoadAcc ? ((first.modes & 3) == kModeVar ? x[first.a] : first.c) : point_term(first, x);
  // -0 adds nothing; the next 32 terms are formed while the last are added
  auto form = [&](int pc) { return pc < pc1 ? point_term(load_instr(prog, pc), x) : -0.0; };
  double p = form(pc0 + 1 + lane);
  for (int base = pc0 + 1; base < pc1; base += 32) {
    const double pn = form(base + 32 + lane);
#pragma unroll
    for (int j = 0; j < 32; ++j) acc = __dadd_rn(acc, __shfl_sync(0xffffffffu, p, j));
    p = pn;
  }
  return acc;
}

// A chain's FP32 value at the point x, one round-to-nearest operation per DAG
// node in program order.
__device__ __forceinline__ float point_chain32(const ChainTerm* __restrict__ term, int t0, int t1,
                                               const float* __restrict__ x, int stride)
{
  const uint2* __restrict__ w = reinterpret_cast<const uint2*>(term);
  float acc = 0.0f;
#pragma unroll 4
  for (int q = t0; q < t1; ++q) {
    const uint2 t = __ldg(w + q);
    const float p = __fmul_rn(x[(int)(t.x & 0xffffu) * stride], x[(int)(t.x >> 16) * stride]);
    acc = __fadd_rn(acc, __fmul_rn(__uint_as_float(t.y), p));
  }
  return acc;
}

// A warp's tile of points, lane < 2^log_pts its point p when cand.  Every
// point that may be the best (or, solver, below the incumbent) is evaluated
// in FP64 and handed to accept(point, value) by one lane; *best_key holds the
// lb_key of the smallest value known so far.
template <class F>
__device__ __forceinline__ void sample_tile(const SampleArgs& a, double* x64, float* x32, uint8_t* list, int log_pts,
                                            const PointOf& p, bool cand, unsigned long long* best_key, double gub,
                                            unsigned long long& rejected, const F& accept)
{
  const int pts = 1 << log_pts, stride = point_stride(log_pts);
  const int lane = threadIdx.x & 31, n = a.n_vars;
  const bool solver = a.state != nullptr;
  const ChainSeg* seg = a.chain.seg;
  const unsigned live = __ballot_sync(0xffffffffu, cand);
  if (live == 0u) return;
  // (1) the points, cut to FP32; few points: their lanes share the draws
  bool bad = false;
  {
    const int pt = lane & (pts - 1), L = 32 >> log_pts;
    PointOf q = p;
    if (L > 1) {
      q.k = __shfl_sync(0xffffffffu, p.k, pt);
      q.r = __shfl_sync(0xffffffffu, p.r, pt);
      q.i = __shfl_sync(0xffffffffu, p.i, pt);
      q.salt = __shfl_sync(0xffffffffu, p.salt, pt);
      q.count = __shfl_sync(0xffffffffu, p.count, pt);
      q.fathom = __shfl_sync(0xffffffffu, (int)p.fathom, pt) != 0;
      q.sp = a.pinfo != nullptr ? a.slots + q.k * (uint64_t)a.max_slots : nullptr;
    }
    if ((live >> pt) & 1u)
      for (int v = lane >> log_pts; v < n; v += L) x32[v * stride + pt] = cut32(coordinate(a, q, v), bad);
  }
  unsigned bad_m = __ballot_sync(0xffffffffu, bad);
  for (int off = pts; off < 32; off <<= 1) bad_m |= bad_m >> off;
  // (2) the constraints, until no point is left
  unsigned cand_m = live, proven_m = live & ~bad_m;
  unsigned alive = live & ~bad_m, dealt = 0;
  Deal d = {};
  for (int q = 1; q < a.chain.n_seg && alive != 0u; ++q) {
    const ChainSeg& s = seg[q];
    if (dealt != alive) d = deal(dealt = alive, list);
    float sum = 0.0f, mag = 0.0f;
    if (d.pt >= 0) filter_point(s, a.chain.term, x32 + d.pt, (uint32_t)stride, d.sub, 1 << d.lg, sum, mag);
    for (int off = 1; off < (1 << d.lg); off <<= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, off);
      mag += __shfl_xor_sync(0xffffffffu, mag, off);
    }
    const float err = s.eps * mag;
    const float lo = __fsub_rd(sum, err), hi = __fadd_ru(sum, err);
    bool out, sure;
    if (s.kind == kChainLe) {
      out = lo > s.rhs_up;
      sure = hi <= s.rhs_dn;
    } else {  // almost_equal's tolerance, at its largest over [lo, hi]
      const float most = fmaxf(fmaxf(fabsf(lo), fabsf(hi)), fmaxf(fabsf(s.rhs_dn), fabsf(s.rhs_up)));
      const float tol = fmaxf(1.001e-8f, 1.001e-6f * most);
      out = __fsub_rd(lo, s.rhs_up) > tol || __fsub_rd(s.rhs_dn, hi) > tol;
      sure = false;
    }
    const bool lead = d.pt >= 0 && d.sub == 0;
    const unsigned bit = lead ? 1u << d.pt : 0u;
    const unsigned out_m = __reduce_or_sync(0xffffffffu, lead && out ? bit : 0u);
    proven_m &= ~__reduce_or_sync(0xffffffffu, lead && !sure ? bit : 0u);
    cand_m &= ~out_m;
    alive &= ~out_m;
  }
  // (3) the objective's lower end in FP32
  float low = -INFINITY;
  if (alive != 0u) {
    if (dealt != alive) d = deal(alive, list);
    float sum = 0.0f, mag = 0.0f;
    if (d.pt >= 0) filter_point(seg[0], a.chain.term, x32 + d.pt, (uint32_t)stride, d.sub, 1 << d.lg, sum, mag);
    for (int off = 1; off < (1 << d.lg); off <<= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, off);
      mag += __shfl_xor_sync(0xffffffffu, mag, off);
    }
    const float end = __fsub_rd(sum, seg[0].eps * mag);
    // to the point's own lane
    const float mine = __shfl_sync(0xffffffffu, end, __popc(alive & ((1u << lane) - 1u)) << d.lg);
    if (((alive >> lane) & 1u) && mine == mine) low = mine;
  }
  cand = (cand_m >> lane) & 1u;
  const bool proven = (proven_m >> lane) & 1u;
  const bool always = p.fathom && solver;  // inadmissible exact points are counted
  // (4) the points left, in FP64: with the whole warp one by one, the
  // smallest FP32 bound first; when the first of them leaves many (their
  // bounds too close to tell apart), half as many at once as the tile has,
  // in columns over the FP32 points, which are done with
  const int cols = pts >> 1, lgc = 6 - log_pts;  // columns, log2 of the lanes on each
  bool first = true;
  for (;;) {
    const double lim = key_value(*(volatile unsigned long long*)best_key);
    if (!always && (double)low > lim) cand = false;
    const unsigned m = __ballot_sync(0xffffffffu, cand);
    if (m == 0u) break;
    const bool many = !first && cols > 1 && __popc(m) >= 6;
    first = false;
    int src, step, part;  // this lane's point, and its share of the work on it
    if (many) {
      part = lane & ((1 << lgc) - 1);
      step = 1 << lgc;
      unsigned rest = m;
      for (int q = lane >> lgc; q > 0; --q) rest &= rest - 1u;
      src = __ffs((int)rest) - 1;  // -1: no point for this column
    } else {
      part = lane;
      step = 32;
      float lo_min = cand ? low : INFINITY;
      for (int off = 16; off > 0; off >>= 1) lo_min = fminf(lo_min, __shfl_xor_sync(0xffffffffu, lo_min, off));
      const unsigned at = __ballot_sync(0xffffffffu, cand && low == lo_min);
      src = __ffs((int)(at != 0u ? at : m)) - 1;
    }
    const int from = src < 0 ? lane : src;
    const uint64_t k1 = __shfl_sync(0xffffffffu, p.k, from), r1 = __shfl_sync(0xffffffffu, p.r, from);
    const uint64_t i1 = __shfl_sync(0xffffffffu, p.i, from), salt1 = __shfl_sync(0xffffffffu, p.salt, from);
    const uint32_t c1 = __shfl_sync(0xffffffffu, p.count, from);
    const bool f1 = __shfl_sync(0xffffffffu, (int)p.fathom, from) != 0;
    const bool p1 = __shfl_sync(0xffffffffu, (int)proven, from) != 0;
    const PointOf one = {k1, r1, i1, salt1, a.pinfo != nullptr ? a.slots + k1 * (uint64_t)a.max_slots : nullptr, c1, f1};
    Tile<double> t = {};
    t.lo = many ? reinterpret_cast<double*>(x32) + (lane >> lgc) : x64;
    t.stride = many ? cols : 1;
    __syncwarp();  // the columns' readers of the previous points are done
    if (src >= 0)
      for (int v = part; v < n; v += step) t.lo[v * t.stride] = coordinate(a, one, v);
    __syncwarp();
    double value = INFINITY;
    if (!many && p1) {
      value = point_chain_warp(a.prog, seg[0].pc0, seg[0].pc1, x64);
    } else {
      PointVerdict pv = {INFINITY, true, false};
      if (src >= 0) pv = run_point_lane(a.prog, a.sched, many ? lgc : 5, part, t);
      pv = group_point_verdict(pv, step);
      if (pv.feasible && pv.obj == pv.obj) value = pv.obj;
    }
    if (value != value) value = INFINITY;
    if (src >= 0 && part == 0 && value < INFINITY) {
      bool ok = true;
      if (f1 && solver) {
        for (int v = 0; v < n && ok; ++v) {
          const double x = t.lo[v * t.stride];
          if (!(x >= a.root_lb[v]) || !(x <= a.root_ub[v])) ok = false;
          else if (a.var_kinds[v] != 0 && fabs(__dsub_rn(x, rint(x))) > 1e-6) ok = false;
        }
        if (!ok && value < gub) ++rejected;
      }
      if (ok) {
        accept(one, value);
        atomicMin(best_key, (unsigned long long)lb_key(value));
      }
    }
    // the points evaluated leave the list
    unsigned done = 0;
    if (many) {
      unsigned rest = m;
      for (int q = 0; q < cols && rest != 0u; ++q) rest &= rest - 1u;
      done = m & ~rest;
    } else {
      done = 1u << src;
    }
    if ((done >> lane) & 1u) cand = false;
    __syncwarp();
  }
  __syncwarp();  // the points are restaged next
}

// The lazy form's chunk of children [32c, 32c + 32): the child and sample
// with the smallest FP32 value (ties: the first child, then the first
// sample).  False when no point of the chunk is feasible in FP32.
__device__ __forceinline__ bool chunk_point(const SampleArgs& a, uint64_t c, uint64_t total, uint64_t salt_base, PointOf& p)
{
  float best = INFINITY;
  uint64_t g = 0, i = 0;
  const uint64_t g0 = c << kChunkLog2;
  const uint64_t g1 = total < g0 + (1ULL << kChunkLog2) ? total : g0 + (1ULL << kChunkLog2);
  for (uint64_t x = g0; x < g1; ++x) {
    const Best32 b = a.cbest[x];
    if (b.value < best) {
      best = b.value;
      g = x;
      i = b.i;
    }
  }
  if (!(best < INFINITY)) return false;
  point_child(a, g, salt_base, p);
  p.i = i;
  return true;
}

// The lazy form's sample screen (sample_screen_kernel's results): every
// sampled child's S points in FP32, one round-to-nearest operation per DAG
// node in program order, keeping the smallest value and its sample in
// cbest[g].  A lane runs whole chains, so a point's lanes take different
// constraints at once.
__device__ __forceinline__ void screen_tile(const SampleArgs& a, float* x, uint8_t* list, int log_pts, uint64_t w0,
                                            uint64_t total, uint64_t salt_base)
{
  const int pts = 1 << log_pts, stride = point_stride(log_pts);
  const int lane = threadIdx.x & 31, n = a.n_vars;
  const ChainSeg* seg = a.chain.seg;
  if (lane < pts) x[n * stride + lane] = 1.0f;  // linear terms
  const uint64_t g = (w0 << log_pts) + lane;
  PointOf p = {};
  const bool mine = lane < pts && g < total;
  const bool take = mine && point_child(a, g, salt_base, p);
  Best32 best = {INFINITY, 0};
  const uint64_t S = p.fathom ? 1 : a.S;
  for (uint64_t i = 0; i < a.S; ++i) {
    unsigned alive = __ballot_sync(0xffffffffu, take && i < S);
    if (alive == 0u) break;
    p.i = i;
    const unsigned drawn = alive;
    {
      const int pt = lane & (pts - 1), L = 32 >> log_pts;
      PointOf q = p;
      if (L > 1) {
        q.k = __shfl_sync(0xffffffffu, p.k, pt);
        q.r = __shfl_sync(0xffffffffu, p.r, pt);
        q.salt = __shfl_sync(0xffffffffu, p.salt, pt);
        q.count = __shfl_sync(0xffffffffu, p.count, pt);
        q.fathom = __shfl_sync(0xffffffffu, (int)p.fathom, pt) != 0;
        q.sp = a.pinfo != nullptr ? a.slots + q.k * (uint64_t)a.max_slots : nullptr;
      }
      if ((drawn >> pt) & 1u)
        for (int v = lane >> log_pts; v < n; v += L) x[v * stride + pt] = __double2float_rn(coordinate(a, q, v));
    }
    __syncwarp();
    Deal d = {};
    unsigned dealt = 0;
    for (int q = 1; q < a.chain.n_seg && alive != 0u;) {
      if (dealt != alive) d = deal(dealt = alive, list);
      bool ok = true;
      if (d.pt >= 0 && q + d.sub < a.chain.n_seg) {
        const ChainSeg& s = seg[q + d.sub];
        const float v = point_chain32(a.chain.term_pt, s.pt, s.pt_end, x + d.pt, stride);
        ok = s.kind == kChainLe ? v <= s.rhs_dn : almost_equal((double)v, s.rhs);
      }
      q += 1 << d.lg;
      alive &= ~__reduce_or_sync(0xffffffffu, d.pt >= 0 && !ok ? 1u << d.pt : 0u);
    }
    if (alive != 0u) {
      float v = INFINITY;
      if ((alive >> lane) & 1u) v = point_chain32(a.chain.term_pt, seg[0].pt, seg[0].pt_end, x + lane, stride);
      if (v < best.value) best = Best32{v, (uint32_t)i};
    }
    __syncwarp();  // the points are restaged next
  }
  if (mine) a.cbest[g] = best;
}

}  // namespace cmn
