// chain_tiles.cuh -- the FP64 evaluator of programs that are sets of sum
// chains (every quadratic model), in two passes: the constraints, a tile of
// boxes per block and a warp per chain; then the objective (chain_core.cuh).
// The single-instance kernels are in chain_kernels.cu, the batch's in
// batch_chain_kernels.cu.
//
// What bounds it: FP64 instructions issue at 1/64 of the FP32 rate, and the
// interpreter spends four of them per term on both bounds of every chain.
// Here the constraints, nine tenths of a program's terms, are decided in
// FP32, and FP64 work is left to the objective's lower bound and to the few
// comparisons the FP32 error bound leaves open.  On the n = 64 MIQCQP (2^17
// regions of one box) the interpreter took 18.5 ms, these passes 0.74 and
// 0.33 ms: the first at 92 % of the shared-memory bandwidth (two 8-byte loads
// per term and box), the second at 68 % of the FP64 pipe.
#pragma once

#include <cfloat>
#include <cstdint>

#include "chain_core.cuh"
#include "child_core.cuh"

namespace cmn {

constexpr int kTileWarps = 8;     // warps of a constraint tile: one per chain below that
constexpr int kObjThreads = 128;  // threads of an objective block

using V64 = ChildVars<double, double>;

// The two-sided interpreter over one chain and its readers.
template <bool kFused>
static __device__ __noinline__ void chain_general(const Instr* prog, int pc0, int pc1, const V64& vars, Verdict<double>& v)
{
  const Tile<double> t = {};
  interval_range<double, V64, kFused>(prog, pc0, pc1, vars, t, v);
}

// A <= chain in FP64: its lower bound against the right side.
template <bool kFused>
static __device__ __noinline__ bool chain_le_exact(const Instr* prog, const ChainSeg& s, const V64& vars)
{
  const double lo = chain_lo<kFused>(prog, s.pc0, s.pc1, vars);
  if (lo == lo) return lo <= s.rhs;
  Verdict<double> v = verdict_init<double>();
  chain_general<kFused>(prog, s.pc0, s.pc2, vars, v);
  return v.feasible;
}

// A constraint tile in shared memory: bounds cut to FP32 and their largest
// magnitudes per variable, and the split variables of each box in FP64.
struct TileSmem {
  float2* x;     // [n_vars][boxes]
  double* olo;   // [max_slots][boxes]
  double* ohi;
  float* hull;   // [n_vars]
  int32_t* ovid;
};

__device__ __forceinline__ TileSmem tile_smem(unsigned char* raw, int n_vars, int ms, int boxes)
{
  TileSmem t;
  t.x = reinterpret_cast<float2*>(raw);
  t.olo = reinterpret_cast<double*>(t.x + (size_t)n_vars * boxes);
  t.ohi = t.olo + (size_t)ms * boxes;
  t.hull = reinterpret_cast<float*>(t.ohi + (size_t)ms * boxes);
  t.ovid = reinterpret_cast<int32_t*>(t.hull + n_vars);
  return t;
}

inline size_t tile_smem_bytes(int n_vars, int ms, int boxes)
{
  return ((size_t)n_vars * 8 + (size_t)ms * 20) * (size_t)boxes + (size_t)n_vars * 4;
}

__device__ __forceinline__ uint64_t box_count(const EvalArgs& a, bool list)
{
  return list ? *a.list_count : (a.n_children_dev ? *a.n_children_dev : a.n_children);
}

__device__ __forceinline__ float max_abs_group(float m, int boxes)
{
  for (int off = 1; off < boxes; off <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  return m;
}

// The constraints of one tile's boxes (all chains but an objective one).  kMode and
// kFused as eval_children's; out_flag gets 0 / 1 (kMode 0 and 4), or
// kChildNone, kChildDuplicate, kChildInfeasible or kChildEligible (1 and 3).
// A tile has 2^log_boxes boxes, 32 >> log_boxes lanes on each; the whole
// block calls this for the same tile.
struct TileShared {
  unsigned fail;  // boxes a constraint excludes
  unsigned bad;   // boxes outside the filter's range
  int next;       // next chain of the tile
};

template <int kMode, bool kFused>
__device__ void constraints_tile(const EvalArgs& a, unsigned char* smem, TileShared& sh, int log_boxes, uint64_t tile,
                                 uint64_t total)
{
  const int boxes = 1 << log_boxes, L = 32 >> log_boxes;
  const TileSmem t = tile_smem(smem, a.n_vars, a.pinfo != nullptr ? a.max_slots : 0, boxes);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int box = lane & (boxes - 1), sub = lane >> log_boxes;
  const int first = a.chain.seg[0].kind == kChainObjective ? 1 : 0;
  // this lane's box; lanes past the end shadow the last one
  const uint64_t at = (tile << log_boxes) + box;
  bool live = at < total;
  const uint64_t idx = live ? at : total - 1;
  const uint64_t g = kMode == 3 ? (uint64_t)a.list[idx] : idx;
  uint64_t k, r;
  child_of(a.log2C, g, k, r);
  const bool writes = live && wid == 0 && sub == 0;
  uint32_t count = 0;
  const SlotPlan* sp = nullptr;
  if (a.pinfo != nullptr) {
    const ParentInfo pi = a.pinfo[k];
    if ((kMode == 1 || kMode == 3) && (pi.fathom || r >= pi.nreg)) {
      if (kMode == 1 && writes) a.out_flag[g] = kChildNone;
      live = false;
    } else {
      count = pi.count;
      sp = a.slots + k * (uint64_t)a.max_slots;
    }
  }
  // (1) the tile: the parents' bounds, then the split variables
  bool bad = false;
  for (int v0 = wid * L; v0 < a.n_vars; v0 += W * L) {
    const int v = v0 + sub;
    float m = 0.0f;
    if (v < a.n_vars) {
      bool b = false;
      const float lo = cut32(__ldg(a.plo + (uint64_t)v * a.pstride + k), b);
      const float hi = cut32(__ldg(a.phi + (uint64_t)v * a.pstride + k), b);
      t.x[v * boxes + box] = make_float2(lo, hi);
      b = b || lo > hi;  // no interval
      bad = bad || b;
      m = b ? 0.0f : fmaxf(fabsf(lo), fabsf(hi));
    }
    m = max_abs_group(m, boxes);
    if (v < a.n_vars && box == 0) t.hull[v] = m;
  }
  if (threadIdx.x == 0) {
    sh.fail = 0;
    sh.bad = 0;
    sh.next = first;
  }
  __syncthreads();
  V64 cv;
  cv.plo = a.plo + k;
  cv.phi = a.phi + k;
  cv.pstride = a.pstride;
  cv.mask = 0;
  cv.olo = t.olo + box;
  cv.ohi = t.ohi + box;
  cv.ovid = t.ovid + box;
  cv.count = (int)count;
  cv.stride = boxes;
  bool dup = false;
  for (uint32_t j = 0; j < count; ++j) {
    const SlotPlan s = sp[j];
    cv.mask |= 1ULL << (s.vid & 63);
    const bool mine = (int)(j % (uint32_t)(W * L)) == wid * L + sub;
    if (kMode == 1 || kMode == 3 || mine) {
      const uint64_t part = slot_part(r, s);
      if (part >= s.dom) dup = true;
      if (mine) {
        double lo, hi;
        slot_bounds(s, a.plo[(uint64_t)s.vid * a.pstride + k], a.phi[(uint64_t)s.vid * a.pstride + k], part, lo, hi);
        t.olo[j * boxes + box] = lo;
        t.ohi[j * boxes + box] = hi;
        t.ovid[j * boxes + box] = (int32_t)s.vid;
        bool leads = true;  // a variable of two slots takes the first one's part
        for (uint32_t q = 0; q < j; ++q) leads = leads && sp[q].vid != s.vid;
        bad = bad || lo > hi;
        if (leads) t.x[s.vid * boxes + box] = make_float2(cut32(lo, bad), cut32(hi, bad));
      }
    }
  }
  if ((kMode == 1 || kMode == 3) && dup) {
    if (live && wid == 0 && sub == 0) a.out_flag[g] = kChildDuplicate;
    live = false;
  }
  if (bad) atomicOr(&sh.bad, 1u << box);
  const unsigned alive = __ballot_sync(0xffffffffu, live);  // the same in every warp
  __syncthreads();
  if (alive != 0u) {
    const bool in_range = !((sh.bad >> box) & 1u);
    // (2) the chains, drawn from a ticket
    for (;;) {
      int q = 0;
      if (lane == 0) q = atomicAdd(&sh.next, 1);
      q = __shfl_sync(0xffffffffu, q, 0);
      if (q >= a.chain.n_seg) break;
      const ChainSeg& s = a.chain.seg[q];
      bool ok = true, open = live && sub == 0;
      if (s.kind == kChainLe && s.eps > 0.0f) {
        const float err = s.eps * chain_magnitude(s, a.chain.term, t.hull);
        float est = filter_chain(s, a.chain.term, t.x + box, (uint32_t)boxes, sub, L);
        for (int off = boxes; off < 32; off <<= 1) est += __shfl_xor_sync(0xffffffffu, est, off);
        if (in_range) {
          ok = !(__fsub_rd(est, err) > s.rhs_up);
          open = open && ok && !(__fadd_ru(est, err) <= s.rhs_dn);
        }
        if (open) ok = chain_le_exact<kFused>(a.prog, s, cv);
      } else if (s.kind == kChainLe) {
        if (open) ok = chain_le_exact<kFused>(a.prog, s, cv);
      } else if (open) {
        Verdict<double> v = verdict_init<double>();
        chain_general<kFused>(a.prog, s.pc0, s.pc2, cv, v);
        ok = v.feasible;
      }
      const unsigned no = __ballot_sync(0xffffffffu, live && sub == 0 && !ok);
      if (lane == 0 && no) atomicOr(&sh.fail, no);
    }
  }
  __syncthreads();
  if (live && wid == 0 && sub == 0) {
    const bool feasible = !((sh.fail >> box) & 1u);
    if (kMode == 0 && a.flags != nullptr) a.flags[g] = feasible ? 1 : 0;
    else if (kMode == 0 || kMode == 4) a.out_flag[g] = feasible ? 1 : 0;
    else a.out_flag[g] = feasible ? kChildEligible : kChildInfeasible;
  }
  __syncthreads();  // the tile is restaged next
}

// ---- the objective of children, a warp per 32 consecutive ones ----
// Siblings share most of their box: a term whose variables no sibling of the
// warp narrows has one value for all of them, and one that reads a slot of
// two parts has two.  Per chunk of 32 terms the warp's lanes form the
// distinct (family, term, parts) values -- a family is the warp's children
// of one parent --, leave them in shared memory, and every lane then adds
// its own in program order.  FP64 work per term and child falls from about
// 3.5 operations to the one add and a few hundredths; the chain of adds is
// the reference's, so the bounds are too.
constexpr int kFamSlots = 5;   // varying slots a family tabulates (32 children vary five bits)
constexpr int kFamWidth = 4;   // widest slot it tabulates; wider ones are computed per child
constexpr int kFamNone = 7;    // descriptor: the variable does not vary

struct Family {
  uint64_t k;
  uint64_t mask;              // ChildVars::mask of its lead lane
  uint64_t wide;              // variables (v & 63) computed per child
  int32_t count;
  int32_t lead;               // its first lane
  int32_t nv;                 // tabulated slots
  int32_t vid[kFamSlots];
  int32_t slot[kFamSlots];
  uint32_t widths;            // 4 bits each
  uint8_t rep[kFamSlots][kFamWidth];  // a lane on each part
};

// A family's box with the variables of one term over given parts.
struct FamVars {
  V64 base;
  int va, vb;  // -1: from base
  Iv<double> a, b;
  __device__ __forceinline__ Iv<double> var(int v) const
  {
    if (v == va) return a;
    if (v == vb) return b;
    return base.var(v);
  }
};

// Most values a chunk needs: 32 terms of up to four each per family, two
// where the families are pairs of children.
inline __host__ __device__ size_t family_values(int families) { return 128 * (size_t)(families < 8 ? families : 8); }
// Bytes of a warp's tables: the values and their items, the descriptors, the
// families, and the children's split variables.
inline __host__ __device__ size_t family_bytes(int families, int ms, bool hi)
{
  return (family_values(families) * (hi ? 18 : 10) + (size_t)families * (32 * 4 + sizeof(Family)) +
          (size_t)ms * 32 * 20 + 15) & ~(size_t)15;
}

// 32 children of one warp; `smem` is its share (family_bytes).
// kTeam: of a block of kTeamWarps.  A chunk's values are latency (12,000 cycles
// with one warp on an SM), so each warp forms those of its own chunk, with
// tables of its own, and the first warp then adds them in order.  `smem` is the
// block's.  The bound phase at n = 32, 4,096 children: 158 -> 99 us; 16,384
// children (four blocks an SM): 193 -> 145 us.
constexpr int kTeamWarps = kObjThreads / 32;
template <int kMode, bool kHi, bool kTeam = false>
__device__ void siblings_tile(const EvalArgs& a, unsigned char* smem, int flags, int families, uint64_t tile,
                              uint64_t total)
{
  const int lane = threadIdx.x & 31, wid = kTeam ? threadIdx.x >> 5 : 0;
  const size_t share = family_bytes(families, a.max_slots, kHi);
  smem += share * wid;
  const int ms = a.max_slots;
  const size_t nval = family_values(families);
  double* vlo = reinterpret_cast<double*>(smem);
  double* vhi = vlo + (kHi ? nval : 0);
  double* olo = vlo + (kHi ? 2 : 1) * nval + lane;
  double* ohi = olo + (size_t)ms * 32;
  Family* fam = reinterpret_cast<Family*>(ohi - lane + (size_t)ms * 32);
  int32_t* ovid = reinterpret_cast<int32_t*>(fam + families) + lane;
  uint32_t* desc = reinterpret_cast<uint32_t*>(ovid - lane + (size_t)ms * 32);
  uint16_t* item = reinterpret_cast<uint16_t*>(desc + (size_t)families * 32);
  const double gub = a.gub ? *a.gub : DBL_MAX;
  const ChainSeg s = a.chain.seg[0];
  const int flanes = 32 / families;  // lanes of a family
  const int f = lane / flanes, lead = f * flanes;
  const unsigned fmask = (flanes == 32 ? 0xffffffffu : ((1u << flanes) - 1u)) << lead;
  const uint64_t at = (tile << 5) + lane;
  bool live = at < total;
  const uint64_t g = live ? at : total - 1;  // lanes past the end shadow the last child
  uint64_t k, r;
  child_of(a.log2C, g, k, r);
  bool feasible = true;
  const ParentInfo pi = a.pinfo[k];
  if (flags && live) {
    const uint8_t fl = kMode == 0 && a.flags != nullptr ? a.flags[g] : a.out_flag[g];
    if (kMode == 1) live = fl == kChildEligible;
    else if (kMode == 4) live = fl != 0;
    feasible = fl != 0;
  } else if (live && kMode == 1 && (pi.fathom || r >= pi.nreg)) {
    a.out_flag[g] = kChildNone;
    live = false;
  }
  if (!__any_sync(0xffffffffu, live)) return;
  bool dup;
  const V64 cv = child_vars<double, double>(a, a.plo, a.phi, k, r, olo, ohi, ovid, 32, dup);
  if (kMode == 1 && !flags && dup) {
    if (live) a.out_flag[g] = kChildDuplicate;
    live = false;
  }
  // the family's varying slots; every lane of it finds the same ones
  const SlotPlan* sp = a.slots + k * (uint64_t)a.max_slots;
  uint32_t parts = 0, widths = 0;
  int nv = 0;
  uint64_t wide = 0;
  if (lane == lead) {
    fam[f].k = k;
    fam[f].mask = cv.mask;
    fam[f].count = cv.count;
    fam[f].lead = lead;
    // parts no child of the warp is on stand for the lead's
    for (int e = 0; e < kFamSlots; ++e)
      for (int q = 0; q < kFamWidth; ++q) fam[f].rep[e][q] = (uint8_t)lead;
  }
  __syncwarp();
  const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)cv.count);
  for (int j = 0; j < most; ++j) {
    const bool has = j < cv.count;
    uint64_t part = 0, width = 1;
    int vid = -1;
    bool first = has;
    if (has) {
      part = slot_part(r, sp[j]);
      width = sp[j].width;
      vid = (int)sp[j].vid;
      for (int q = 0; q < j; ++q) first = first && ovid[q * 32] != vid;  // ChildVars reads the first slot
    }
    const uint64_t p0 = __shfl_sync(0xffffffffu, part, lead);
    const bool varies = (__ballot_sync(0xffffffffu, first && part != p0) & fmask) != 0u;
    if (varies) {
      if (width <= kFamWidth && nv < kFamSlots) {
        if (lane == lead) {
          fam[f].vid[nv] = vid;
          fam[f].slot[nv] = j;
        }
        fam[f].rep[nv][part] = (uint8_t)lane;  // any lane on that part will do
        parts |= (uint32_t)part << (4 * nv);
        widths |= (uint32_t)width << (4 * nv);
        ++nv;
      } else {
        wide |= 1ULL << (vid & 63);
      }
    }
  }
  if (lane == lead) {
    fam[f].nv = nv;
    fam[f].widths = widths;
    fam[f].wide = wide;
  }
  __syncwarp();
  double lo = 0.0, hi = 0.0;
  constexpr int kRound = kTeam ? 32 * kTeamWarps : 32;
  for (int round = s.pc0; round < s.pc1; round += kRound) {
    const int base = round + 32 * wid, left = s.pc1 - base;
    const int cnt = left < 32 ? (left < 0 ? 0 : left) : 32;
    // (1) lane = term: how many values each family needs, and where
    int filled = 0;
    bool any_wide = false;
    Instr cur = {};
    if (lane < cnt) cur = load_instr(a.prog, base + lane);
    const int code = cur.head & 7, pk = (cur.head >> 3) & kTermPMask;
    const bool reads_a = code == kOpTerm || (cur.modes & 3) == kModeVar;
    const bool reads_b = code == kOpTerm && pk == kTermProd && cur.b != cur.a;
    for (int q = 0; q < families; ++q) {
      const Family& F = fam[q];
      int ca = kFamNone, cb = kFamNone, wa = 1, wb = 1;
      bool per_child = false;
      if (lane < cnt) {
        for (int e = 0; e < F.nv; ++e) {
          const int w = (int)(F.widths >> (4 * e)) & 15;
          if (reads_a && F.vid[e] == cur.a) ca = e, wa = w;
          if (reads_b && F.vid[e] == cur.b) cb = e, wb = w;
        }
        per_child = (reads_a && ((F.wide >> (cur.a & 63)) & 1)) || (reads_b && ((F.wide >> (cur.b & 63)) & 1));
      }
      // a product of two four-part slots would outgrow the table
      per_child = per_child || wa * wb > kFamWidth;
      const int need = lane < cnt && !per_child ? wa * wb : 0;
      int x = need;
      for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
      }
      const int pos = filled + x - need;
      if (lane < cnt)
        desc[q * 32 + lane] = (uint32_t)pos | (uint32_t)ca << 16 | (uint32_t)cb << 20 | (uint32_t)wa << 24 | (per_child ? 1u << 31 : 0u);
      for (int e = 0; e < need; ++e) item[pos + e] = (uint16_t)(q << 7 | lane << 2 | e);
      filled += __shfl_sync(0xffffffffu, x, 31);
      any_wide = any_wide || __any_sync(0xffffffffu, per_child);
    }
    __syncwarp();
    // (2) lane = value
    for (int it = lane; it < filled; it += 32) {
      const uint32_t code_it = item[it];
      const int q = (int)(code_it >> 7), j = (int)(code_it >> 2) & 31, combo = (int)code_it & 3;
      const Family& F = fam[q];
      const uint32_t d = desc[q * 32 + j];
      const int ca = (int)(d >> 16) & 15, cb = (int)(d >> 20) & 15, wa = (int)(d >> 24) & 15;
      const Instr ins = load_instr(a.prog, base + j);
      FamVars fv;
      fv.base.plo = a.plo + F.k;
      fv.base.phi = a.phi + F.k;
      fv.base.pstride = a.pstride;
      fv.base.mask = F.mask;
      fv.base.olo = olo - lane + F.lead;
      fv.base.ohi = ohi - lane + F.lead;
      fv.base.ovid = ovid - lane + F.lead;
      fv.base.count = F.count;
      fv.base.stride = 32;
      fv.va = fv.vb = -1;
      if (ca != kFamNone) {
        const int rl = F.rep[ca][combo % wa] - lane, o = F.slot[ca] * 32 + rl;
        fv.va = ins.a;
        fv.a = Iv<double>{olo[o], ohi[o]};
      }
      if (cb != kFamNone) {
        const int rl = F.rep[cb][combo / wa] - lane, o = F.slot[cb] * 32 + rl;
        fv.vb = ins.b;
        fv.b = Iv<double>{olo[o], ohi[o]};
      }
      const int sub = ins.head >> 3;
      const bool neg = (sub & kTermSub) != 0 && !(sub & kTermInit);
      if ((ins.head & 7) == kOpLoadAcc) {
        const Iv<double> x = (ins.modes & 3) == kModeVar ? fv.var(ins.a) : Iv<double>{ins.c, ins.c};
        vlo[it] = x.lo;
        if (kHi) vhi[it] = x.hi;
      } else {
        const double l = term_lo<false>(ins, fv);
        vlo[it] = neg ? -l : l;
        if (kHi) {
          const double h = term_hi(ins, fv);
          vhi[it] = neg ? -h : h;
        }
      }
    }
    // (3) lane = child: its terms in order
    auto add_chunk = [&](int base, int cnt, const uint32_t* dl, const double* vlo, const double* vhi, bool any_wide) {
      auto value_at = [&](uint32_t d) {
        const uint32_t pa = (parts >> (4 * ((d >> 16) & 7))) & 15u, pb = (parts >> (4 * ((d >> 20) & 7))) & 15u;
        return (d & 0xffffu) + pa + pb * ((d >> 24) & 15u);
      };
      auto add = [&](int j, double l, double h) {
        const bool start = base + j == s.pc0;
        lo = start ? l : __dadd_rd(lo, l);
        if (kHi) hi = start ? h : __dadd_ru(hi, h);
      };
      if (!any_wide) {
#pragma unroll 8
        for (int j = 0; j < cnt; ++j) {
          const uint32_t at_v = value_at(dl[j]);
          add(j, vlo[at_v], kHi ? vhi[at_v] : 0.0);
        }
      } else {
        for (int j = 0; j < cnt; ++j) {
          const uint32_t d = dl[j];
          double l, h = 0.0;
          if (d >> 31) {
            const Instr ins = load_instr(a.prog, base + j);
            const int sub = ins.head >> 3;
            const bool neg = (sub & kTermSub) != 0 && !(sub & kTermInit);
            if ((ins.head & 7) == kOpLoadAcc) {
              const Iv<double> x = cv.var(ins.a);
              l = x.lo;
              h = x.hi;
            } else {
              l = term_lo<false>(ins, cv);
              l = neg ? -l : l;
              if (kHi) {
                h = term_hi(ins, cv);
                h = neg ? -h : h;
              }
            }
          } else {
            const uint32_t at_v = value_at(d);
            l = vlo[at_v];
            if (kHi) h = vhi[at_v];
          }
          add(j, l, h);
        }
      }
    };
    if constexpr (kTeam) {
      __shared__ int wide_s[kTeamWarps];
      if (lane == 0) wide_s[wid] = any_wide;
      __syncthreads();
      for (int q = 0; wid == 0 && q < kTeamWarps && round + 32 * q < s.pc1; ++q) {
        const int at = round + 32 * q, in = s.pc1 - at < 32 ? s.pc1 - at : 32;
        auto of = [&](auto* p) { return reinterpret_cast<decltype(p)>(reinterpret_cast<unsigned char*>(p) + share * q); };
        add_chunk(at, in, of(desc) + f * 32, of(vlo), of(vhi), wide_s[q] != 0);
      }
      __syncthreads();  // the tables are refilled next
    } else {
      __syncwarp();
      add_chunk(base, cnt, desc + f * 32, vlo, vhi, any_wide);
    }
    __syncwarp();  // the tables are refilled next
  }
  if (wid != 0) return;
  Verdict<double> v = verdict_init<double>();
  v.obj.lo = lo;
  v.obj.hi = hi;
  if (live && (lo != lo || (kHi && hi != hi))) chain_general<false>(a.prog, s.pc0, s.pc2, cv, v);
  v.feasible = feasible;
  if constexpr (kMode == 4) {
    aggregate_fold(a, live, r, v);
  } else {
    if (live) write_verdict<double, kMode>(a, g, k, v, gub);
  }
  __syncwarp();  // the columns are rewritten next
}

}  // namespace cmn
