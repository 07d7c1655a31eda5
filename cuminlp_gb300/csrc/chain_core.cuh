// chain_core.cuh -- device arithmetic of sum-chain programs (Program::chain_*):
// one warp evaluates one chain for 32 boxes, lane = box.
//
// A verdict needs one bound of each chain: a <= constraint compares its
// chain's lower bound with the right side, the search orders boxes by the
// objective's lower bound.  So the chains here carry the lower bound alone
// (the objective's upper bound where a caller asks for it), with exactly the
// roundings the two-sided interpreter gives that bound.
//
// A <= constraint is decided in FP32 first.  The FP32 chain sums the same
// terms over bounds cut to FP32, in any order; the FP64 lower bound lies
// within ChainSeg::eps * M of it, M the sum of the terms' largest magnitudes
// over the tile (chain_eps in program.cpp).  When that interval does not
// contain the right side, the FP64 comparison is known; otherwise the chain
// is evaluated in FP64.  The decision is the FP64 one either way.
#pragma once

#include <cstdint>

#include "eval_core.cuh"
#include "kernels.cuh"

namespace cmn {

// A double cut to FP32 towards zero, on the integer pipe (the conversion
// instruction issues at the FP64 rate).  Exact for +-0; for magnitudes in
// [2^-40, 2^40] the relative error is below 2^-23.  Anything else sets `bad`.
__device__ __forceinline__ float cut32(double x, bool& bad)
{
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mag = hi & 0x7fffffffu;
  const bool zero = (mag | lo) == 0u;
  // biased exponent of 2^-40 is 983, of 2^40 1063
  bad = bad || (!zero && (mag - (983u << 20) >= (80u << 20)));
  const uint32_t m = __funnelshift_l(lo, mag, 3) - ((1023u - 127u) << 23);
  return __uint_as_float((hi & 0x80000000u) | (zero ? 0u : m));
}

// ---- FP32 lower bound of one chain ----
__device__ __forceinline__ float min4(float a, float b, float c, float d) { return fminf(fminf(fminf(a, b), c), d); }
__device__ __forceinline__ float max4(float a, float b, float c, float d) { return fmaxf(fmaxf(fmaxf(a, b), c), d); }

// Terms [q0, q1) of one group, two per 16-byte load; the lanes `sub` of the
// L that share a box take every L-th pair.
template <class F>
__device__ __forceinline__ void filter_group(const ChainTerm* __restrict__ term, int q0, int q1, int sub, int L, const F& f)
{
  const uint4* __restrict__ w = reinterpret_cast<const uint4*>(term);
#pragma unroll 2
  for (int q = (q0 >> 1) + sub; q < (q1 >> 1); q += L) {
    const uint4 t = __ldg(w + q);
    f(0, t.x & 0xffffu, t.x >> 16, __uint_as_float(t.y));
    f(1, t.z & 0xffffu, t.z >> 16, __uint_as_float(t.w));
  }
}

// This lane's share of the chain's lower bound over the box at x (one float2
// of cut bounds per variable, `stride` apart).  Any order of the terms will
// do: chain_eps bounds the error of every grouping.
__device__ __forceinline__ float filter_chain(const ChainSeg& s, const ChainTerm* __restrict__ term,
                                              const float2* __restrict__ x, uint32_t stride, int sub, int L)
{
  float acc[2] = {sub == 0 ? s.c0 : 0.0f, 0.0f};
  filter_group(term, s.group[0], s.group[1], sub, L, [&](int u, uint32_t a, uint32_t b, float c) {  // c > 0, x_a * x_b
    const float2 p = x[a * stride], q = x[b * stride];
    acc[u] = __fmaf_rn(c, min4(p.x * q.x, p.x * q.y, p.y * q.x, p.y * q.y), acc[u]);
  });
  filter_group(term, s.group[1], s.group[2], sub, L, [&](int u, uint32_t a, uint32_t b, float c) {  // c < 0, x_a * x_b
    const float2 p = x[a * stride], q = x[b * stride];
    acc[u] = __fmaf_rn(c, max4(p.x * q.x, p.x * q.y, p.y * q.x, p.y * q.y), acc[u]);
  });
  filter_group(term, s.group[2], s.group[3], sub, L, [&](int u, uint32_t a, uint32_t, float c) {  // c > 0, sqr(x_a)
    const float2 p = x[a * stride];
    const float d = fmaxf(fmaxf(p.x, -p.y), 0.0f);
    acc[u] = __fmaf_rn(c, d * d, acc[u]);
  });
  filter_group(term, s.group[3], s.group[4], sub, L, [&](int u, uint32_t a, uint32_t, float c) {  // c < 0, sqr(x_a)
    const float2 p = x[a * stride];
    const float d = fmaxf(-p.x, p.y);
    acc[u] = __fmaf_rn(c, d * d, acc[u]);
  });
  filter_group(term, s.group[4], s.group[5], sub, L, [&](int u, uint32_t a, uint32_t, float c) {
    acc[u] = __fmaf_rn(c, x[a * stride].x, acc[u]);
  });
  filter_group(term, s.group[5], s.group[6], sub, L, [&](int u, uint32_t a, uint32_t, float c) {
    acc[u] = __fmaf_rn(c, x[a * stride].y, acc[u]);
  });
  return acc[0] + acc[1];
}

// Summed magnitude of the chain's terms over boxes whose variables stay
// within [-hull[v], hull[v]]; the whole warp, the sum in every lane.
__device__ __forceinline__ float chain_magnitude(const ChainSeg& s, const ChainTerm* __restrict__ term,
                                                 const float* __restrict__ hull)
{
  const int lane = threadIdx.x & 31;
  float m = lane == 0 ? fabsf(s.c0) : 0.0f;
  for (int q = s.group[0] + lane; q < s.group[6]; q += 32) {
    const ChainTerm t = term[q];
    const float xa = hull[t.ab & 0xffffu];
    m = __fmaf_rn(fabsf(t.c) * xa, q < s.group[4] ? hull[t.ab >> 16] : 1.0f, m);
  }
  for (int off = 16; off > 0; off >>= 1) m += __shfl_xor_sync(0xffffffffu, m, off);
  return m;
}

// ---- FP64 lower bound of one chain ----
// The lower (upper) end of iv_mul, except that a NaN among the two products
// of operands that both straddle zero always wins; chain_lo's callers look
// for a NaN result and take the interpreter's for it.
__device__ __forceinline__ uint64_t mag_bits(double x) { return (uint64_t)__double_as_longlong(x) & 0x7fffffffffffffffULL; }

__device__ __forceinline__ double mul_lo(Iv<double> a, Iv<double> b)
{
  using A = Arith<double>;
  const bool ap = !A::sgn(a.lo), an = A::sgn(a.hi), bp = !A::sgn(b.lo), bn = A::sgn(b.hi);
  const double la = ap ? (bp ? a.lo : a.hi) : (an ? (bn ? a.hi : a.lo) : (bn ? a.hi : a.lo));
  const double lb = ap ? b.lo : (an ? b.hi : (bn ? b.lo : b.hi));
  double r = emul_rd(la, lb);
  if (!ap && !an && !bp && !bn) {
    // both products are <= 0: the smaller has the larger magnitude
    const double l2 = emul_rd(a.hi, b.lo);
    r = mag_bits(l2) > mag_bits(r) ? l2 : r;
  }
  return r;
}

__device__ __forceinline__ double mul_hi(Iv<double> a, Iv<double> b)
{
  using A = Arith<double>;
  const bool ap = !A::sgn(a.lo), an = A::sgn(a.hi), bp = !A::sgn(b.lo), bn = A::sgn(b.hi);
  const double ua = ap ? (bn ? a.lo : a.hi) : (an ? (bp ? a.hi : a.lo) : (bn ? a.lo : a.hi));
  const double ub = ap ? b.hi : (an ? b.lo : (bn ? b.lo : b.hi));
  double r = emul_ru_sel<double, true>(ua, ub);
  if (!ap && !an && !bp && !bn) {
    // both products are >= 0
    const double u2 = emul_ru_sel<double, true>(a.lo, b.lo);
    r = mag_bits(u2) > mag_bits(r) ? u2 : r;
  }
  return r;
}

// The end of x_a * x_b, sqr(x_a) or x_a that the chain's lower bound reads:
// the lower one for a positive coefficient, the upper one for a negative.
template <typename V>
__device__ __forceinline__ double product_end(const Instr& cur, int sub, bool upper, const V& vars)
{
  const int pk = sub & kTermPMask;
  if (pk == kTermProd) {
    const Iv<double> a = vars.var(cur.a), b = vars.var(cur.b);
    return upper ? mul_hi(a, b) : mul_lo(a, b);
  }
  const Iv<double> a = vars.var(cur.a);
  if (pk == kTermSqr) {
    const Iv<double> s = iv_sqr<double, true>(a);
    return upper ? s.hi : s.lo;
  }
  return upper ? a.hi : a.lo;
}

// One term's operand of the chain's lower bound.  Plain: the bound of the
// whole term that is added (or, kTermSub, subtracted).  Fused: the product
// end that term_apply_lo folds in with one FMA.
template <bool kFused, typename V>
__device__ __forceinline__ double term_lo(const Instr& cur, const V& vars)
{
  using A = Arith<double>;
  const int sub = cur.head >> 3;
  const bool has_c = (sub & kTermHasC) != 0;
  const bool neg = (sub & kTermSub) != 0 && !(sub & kTermInit);
  if (fused_term<double, kFused>(sub)) {
    const double cc = neg ? -cur.c : cur.c;
    return product_end(cur, sub, !(!A::sgn(cc) || A::is_zero(cc)), vars);
  }
  const bool cn = has_c && A::sgn(cur.c);
  const double p = product_end(cur, sub, cn != neg, vars);
  if (!has_c) return p;
  return neg ? emul_ru(cur.c, p) : emul_rd(cur.c, p);
}

// The upper bound's operand of a plain chain: the mirror of term_lo.
template <typename V>
__device__ __forceinline__ double term_hi(const Instr& cur, const V& vars)
{
  using A = Arith<double>;
  const int sub = cur.head >> 3;
  const bool has_c = (sub & kTermHasC) != 0;
  const bool neg = (sub & kTermSub) != 0 && !(sub & kTermInit);
  const bool cn = has_c && A::sgn(cur.c);
  const double p = product_end(cur, sub, cn == neg, vars);
  if (!has_c) return p;
  return neg ? emul_rd(cur.c, p) : emul_ru(cur.c, p);
}

template <bool kFused>
__device__ __forceinline__ double term_apply_lo(double acc, const Instr& cur, double p)
{
  const int sub = cur.head >> 3;
  const bool neg = (sub & kTermSub) != 0;
  if (fused_term<double, kFused>(sub)) return __fma_rd(neg ? -cur.c : cur.c, p, acc);
  if (sub & kTermInit) return p;
  return neg ? __dsub_rd(acc, p) : __dadd_rd(acc, p);
}

// The chain [pc0, pc1): TERMs, the first of which may be a LoadAcc.
template <bool kFused, typename V>
__device__ __forceinline__ double chain_lo(const Instr* __restrict__ prog, int pc0, int pc1, const V& vars)
{
  double acc = 0.0;
  int pc = pc0;
  const Instr first = load_instr(prog, pc);
  if ((first.head & 7) == kOpLoadAcc) {
    acc = (first.modes & 3) == kModeVar ? vars.var(first.a).lo : first.c;
    ++pc;
  }
  // both products of a pair before its first add, so that they overlap
  for (; pc + 2 <= pc1; pc += 2) {
    const Instr c0 = load_instr(prog, pc), c1 = load_instr(prog, pc + 1);
    const double p0 = term_lo<kFused>(c0, vars);
    const double p1 = term_lo<kFused>(c1, vars);
    acc = term_apply_lo<kFused>(acc, c0, p0);
    acc = term_apply_lo<kFused>(acc, c1, p1);
  }
  if (pc < pc1) {
    const Instr c0 = load_instr(prog, pc);
    acc = term_apply_lo<kFused>(acc, c0, term_lo<kFused>(c0, vars));
  }
  return acc;
}

// The same chain by a group of G = 2^kLg lanes on one box: the lanes form G
// terms at once, then every lane adds them in order.  Every lane of the warp
// calls it; a lane without a box passes active = false.  A term past the end
// is +0 times 1, which adds nothing in this rounding; a term that is not
// fused is its value times 1, the same sum.
template <int kLg, bool kFused, typename V>
__device__ __noinline__ double chain_lo_lanes(const Instr* __restrict__ prog, int pc0, int pc1, const V& vars, bool active)
{
  constexpr int G = 1 << kLg;
  const int gl = threadIdx.x & (G - 1);
  double acc = 0.0;
  const Instr first = load_instr(prog, pc0);
  if (active) {
    if ((first.head & 7) == kOpLoadAcc) acc = (first.modes & 3) == kModeVar ? vars.var(first.a).lo : first.c;
    else acc = term_lo<kFused>(first, vars);  // initialising TERM
  }
  // the next G terms are formed while the last ones are added
  auto form = [&](int pc, double& p, double& c) {
    p = 0.0;
    c = 1.0;
    if (!active || pc >= pc1) return;
    const Instr cur = load_instr(prog, pc);
    const int sub = cur.head >> 3;
    const bool neg = (sub & kTermSub) != 0;
    p = term_lo<kFused>(cur, vars);
    if (fused_term<double, kFused>(sub)) c = neg ? -cur.c : cur.c;
    else if (neg) p = -p;
  };
  double p, c;
  form(pc0 + 1 + gl, p, c);
  for (int base = pc0 + 1; base < pc1; base += G) {
    double pn, cn;
    form(base + G + gl, pn, cn);
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const double pj = __shfl_sync(0xffffffffu, p, j, G);
      if (kFused) acc = __fma_rd(__shfl_sync(0xffffffffu, c, j, G), pj, acc);
      else acc = __dadd_rd(acc, pj);
    }
    p = pn;
    c = cn;
  }
  return acc;
}

template <bool kFused, typename V>
__device__ __forceinline__ double chain_lo_group(const Instr* __restrict__ prog, int pc0, int pc1, const V& vars, int lg,
                                                 bool active)
{
  switch (lg) {
    case 1: return chain_lo_lanes<1, kFused>(prog, pc0, pc1, vars, active);
    case 2: return chain_lo_lanes<2, kFused>(prog, pc0, pc1, vars, active);
    case 3: return chain_lo_lanes<3, kFused>(prog, pc0, pc1, vars, active);
    case 4: return chain_lo_lanes<4, kFused>(prog, pc0, pc1, vars, active);
    case 5: return chain_lo_lanes<5, kFused>(prog, pc0, pc1, vars, active);
    default: return active ? chain_lo<kFused>(prog, pc0, pc1, vars) : 0.0;
  }
}

// The upper bound of a plain chain by a group of lanes: the mirror of
// chain_lo_lanes.  A term past the end is -0, which adds nothing in this
// rounding.
template <int kLg, typename V>
__device__ __noinline__ double chain_hi_lanes(const Instr* __restrict__ prog, int pc0, int pc1, const V& vars, bool active)
{
  constexpr int G = 1 << kLg;
  const int gl = threadIdx.x & (G - 1);
  double acc = 0.0;
  const Instr first = load_instr(prog, pc0);
  if (active) {
    if ((first.head & 7) == kOpLoadAcc) acc = (first.modes & 3) == kModeVar ? vars.var(first.a).hi : first.c;
    else acc = term_hi(first, vars);  // initialising TERM
  }
  auto form = [&](int pc) {
    if (!active || pc >= pc1) return -0.0;
    const Instr cur = load_instr(prog, pc);
    const double h = term_hi(cur, vars);
    return ((cur.head >> 3) & kTermSub) != 0 ? -h : h;
  };
  double p = form(pc0 + 1 + gl);
  for (int base = pc0 + 1; base < pc1; base += G) {
    const double pn = form(base + G + gl);
#pragma unroll
    for (int j = 0; j < G; ++j) acc = __dadd_ru(acc, __shfl_sync(0xffffffffu, p, j, G));
    p = pn;
  }
  return acc;
}

template <typename V>
__device__ __forceinline__ double chain_hi_group(const Instr* __restrict__ prog, int pc0, int pc1, const V& vars, int lg,
                                                 bool active)
{
  switch (lg) {
    case 1: return chain_hi_lanes<1>(prog, pc0, pc1, vars, active);
    case 2: return chain_hi_lanes<2>(prog, pc0, pc1, vars, active);
    case 3: return chain_hi_lanes<3>(prog, pc0, pc1, vars, active);
    case 4: return chain_hi_lanes<4>(prog, pc0, pc1, vars, active);
    default: return chain_hi_lanes<5>(prog, pc0, pc1, vars, active);
  }
}

}  // namespace cmn
