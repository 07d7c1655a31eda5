// chain_kernels.cu -- the FP64 evaluator of programs that are sets of sum
// chains, over the boxes of one instance: chain_tiles.cuh's two passes.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "chain_tiles.cuh"
#include "launch.hpp"

namespace cmn {

template <int kMode, bool kFused>
__global__ void __launch_bounds__(kTileWarps * 32, 4) chain_constraints_kernel(const EvalArgs a, int log_boxes)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TileShared sh;
  if (a.done != nullptr && *a.done) return;
  if constexpr (kFused) stamp_first(a.t_first);
  const uint64_t total = box_count(a, kMode == 3);
  const uint64_t tiles = (total + (1ULL << log_boxes) - 1) >> log_boxes;
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x)
    constraints_tile<kMode, kFused>(a, smem_raw, sh, log_boxes, tile, total);
}

// The objective of every box the constraints left (kMode 0: of every box).
// `flags`: the constraint pass ran, out_flag holds its verdicts; otherwise
// no chain decides feasibility and the children's states are found here.
// 2^lg lanes share a box when few boxes are live.
template <int kMode, bool kFused, bool kHi, bool kLanes>
__device__ __forceinline__ void objective_boxes(const EvalArgs& a, unsigned char* smem_raw, int flags, uint64_t total,
                                                unsigned block, unsigned blocks)
{
  const int B = blockDim.x;
  const int ms = a.pinfo != nullptr ? a.max_slots : 0;
  double* olo = reinterpret_cast<double*>(smem_raw) + threadIdx.x;
  double* ohi = olo + (size_t)ms * B;
  int32_t* ovid = reinterpret_cast<int32_t*>(reinterpret_cast<double*>(smem_raw) + (size_t)2 * ms * B) + threadIdx.x;
  const double gub = a.gub ? *a.gub : DBL_MAX;
  const ChainSeg s = a.chain.seg[0];
  const bool pure = s.kind == kChainObjective;
  const int lg = lanes_per_box(total, (uint64_t)blocks * B, pure && (!kHi || kLanes) ? 32 : 1);
  const int G = 1 << lg;
  const uint64_t per_block = (uint64_t)(B >> lg);
  for (uint64_t base = (uint64_t)block * per_block; base < total; base += (uint64_t)blocks * per_block) {
    const uint64_t idx = base + (threadIdx.x >> lg);
    const bool lead = (threadIdx.x & (G - 1)) == 0;
    bool live = idx < total;
    uint64_t g = 0, k = 0, r = 0;
    V64 cv = {};
    bool feasible = true;
    if (live) {
      g = kMode == 3 ? (uint64_t)a.list[idx] : idx;
      child_of(a.log2C, g, k, r);
      if (flags) {
        const uint8_t f = kMode == 0 && a.flags != nullptr ? a.flags[g] : a.out_flag[g];
        if (kMode == 1 || kMode == 3) live = f == kChildEligible;
        else if (kMode == 4 || kFused) live = f != 0;
        feasible = f != 0;
      } else if ((kMode == 1 || kMode == 3) && a.pinfo != nullptr) {
        const ParentInfo pi = a.pinfo[k];
        if (pi.fathom || r >= pi.nreg) {
          if (kMode == 1 && lead) a.out_flag[g] = kChildNone;
          live = false;
        }
      }
    }
    if (live) {
      bool dup;
      cv = child_vars<double, double>(a, a.plo, a.phi, k, r, olo, ohi, ovid, B, dup);
      if (!flags && (kMode == 1 || kMode == 3) && dup) {
        if (lead) a.out_flag[g] = kChildDuplicate;
        live = false;
      }
    }
    Verdict<double> v = verdict_init<double>();
    // (both bounds: one lane a box forms them together in the interpreter)
    bool general = !pure || (kHi && (!kLanes || lg == 0));
    if (!general) {
      v.obj.lo = chain_lo_group<kFused>(a.prog, s.pc0, s.pc1, cv, lg, live);
      general = v.obj.lo != v.obj.lo;
      if constexpr (kHi && kLanes) {
        v.obj.hi = chain_hi_group(a.prog, s.pc0, s.pc1, cv, lg, live);
        general = general || v.obj.hi != v.obj.hi;
      }
    }
    if (general && live) chain_general<kFused>(a.prog, s.pc0, s.pc2, cv, v);
    v.feasible = feasible;
    if constexpr (kMode == 4) {
      aggregate_fold(a, live && lead, r, v);
    } else {
      if (live && lead) write_verdict<double, kMode>(a, g, k, v, gub);
    }
  }
  if constexpr (kFused)
    if ((threadIdx.x & 31) == 0) stamp_last(a.t_last, (uint64_t)block * per_block < total);
}

// kLanes: lane groups for both bounds too.
template <int kMode, bool kFused, bool kHi, bool kLanes = false>
__global__ void __launch_bounds__(kObjThreads, 5) chain_objective_kernel(const EvalArgs a, int flags)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.done != nullptr && *a.done) return;
  if constexpr (kFused)
    if (!flags) stamp_first(a.t_first);
  objective_boxes<kMode, kFused, kHi, kLanes>(a, smem_raw, flags, box_count(a, kMode == 3), blockIdx.x, gridDim.x);
}

// Most children the lane groups above take rather than the sharing kernel
// below, for families of 2^lc consecutive siblings (all of them up to lc = 2).
// With up to 32 lanes a child they cost little more for 512 children than for
// 16; from there the FP64 pipes fill, and sharing the terms' values pays.  The
// bound phase at n = 32, lane groups against sharing: 16 siblings, 512 children
// 73 and 84 us, 1,024 children 99 and 88, 4,096 children 199 and 99; 8 siblings,
// 512 children 72 and 105 us, 2,048 children 144 and 112.  Two or four siblings
// have few values in common and many families to tabulate: n = 12, four
// siblings, 16,384 children 62 and 80 us, 262,144 children 234 and 317.
static __host__ __device__ uint64_t objective_few(int lc) { return lc <= 2 ? ~0ULL : 512; }

template <int kMode, bool kHi>
__global__ void __launch_bounds__(kObjThreads, 5) chain_siblings_kernel(const EvalArgs a, int flags, int families,
                                                                           int few)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.done != nullptr && *a.done) return;
  const int wid = threadIdx.x >> 5, W = blockDim.x >> 5;
  const uint64_t total = box_count(a, false), tiles = (total + 31) >> 5;
  if constexpr (!kHi)
    if (total <= (uint64_t)few) {
      objective_boxes<kMode, false, false, false>(a, smem_raw, flags, total, blockIdx.x, gridDim.x);
      return;
    }
  if (tiles <= gridDim.x) {  // a block for every tile
    if (blockIdx.x < tiles) siblings_tile<kMode, kHi, true>(a, smem_raw, flags, families, blockIdx.x, total);
    return;
  }
  unsigned char* smem = smem_raw + family_bytes(families, a.max_slots, kHi) * wid;
  for (uint64_t tile = (uint64_t)blockIdx.x * W + wid; tile < tiles; tile += (uint64_t)gridDim.x * W)
    siblings_tile<kMode, kHi>(a, smem, flags, families, tile, total);
}

// Both passes of a role's regions in one launch: a region's bound does not wait
// for its feasibility, and with few regions each pass is latency on a part of
// the GPU.  The first `objective` blocks take the objective, the others the
// constraints; `oa` leaves out_flag to them.  A call's time in two launches and
// in one: n = 4, 4 regions 40 and 29 us; n = 32, 4,096 regions 124 and 101;
// n = 64, 8,192 regions 170 and 123.
__global__ void __launch_bounds__(kObjThreads, 5) chain_role_kernel(const EvalArgs ca, const EvalArgs oa, int log_boxes,
                                                                    unsigned objective, int share)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TileShared sh;
  if (blockIdx.x < objective) {
    const uint64_t total = box_count(oa, false);
    if (share) siblings_tile<0, false, true>(oa, smem_raw, 0, 1, blockIdx.x, total);
    else objective_boxes<0, false, false, false>(oa, smem_raw, 0, total, blockIdx.x, objective);
    return;
  }
  const uint64_t total = box_count(ca, false);
  const uint64_t tiles = (total + (1ULL << log_boxes) - 1) >> log_boxes;
  for (uint64_t tile = blockIdx.x - objective; tile < tiles; tile += gridDim.x - objective)
    constraints_tile<0, false>(ca, smem_raw, sh, log_boxes, tile, total);
}

static size_t objective_smem(const EvalArgs& a)
{
  return (size_t)(a.pinfo != nullptr ? a.max_slots : 0) * 20 * kObjThreads;
}

template <int kMode, bool kFused, bool kHi>
static cudaError_t launch_chain_t(const EvalArgs& a, cudaStream_t s)
{
  const int ms = a.pinfo != nullptr ? a.max_slots : 0;
  const int chains = a.chain.n_seg - (a.chain.pure_objective ? 1 : 0);
  if (chains > 0) {
    // smaller tiles, more lanes per box, until the tiles fill the GPU
    int lb = 5;
    while (lb > 0 && (a.max_boxes >> lb) < (uint64_t)sm_count() * 2) --lb;
    auto kernel = chain_constraints_kernel<kMode, kFused>;
    const int threads = 32 * (chains < kTileWarps ? chains : kTileWarps);
    const size_t smem = tile_smem_bytes(a.n_vars, ms, 1 << lb);
    const uint64_t grid = resident_blocks((a.max_boxes + (1ull << lb) - 1) >> lb, kernel, threads, smem);
    kernel<<<(unsigned)grid, threads, smem, s>>>(a, lb);
  }
  if constexpr (!kFused && kMode != 3) {
    // children (of a role's box or of the solver's parents): siblings share
    const int lc = a.log2C < 0 || a.log2C > 5 ? 5 : a.log2C;
    const size_t fsmem = (kObjThreads / 32) * family_bytes(32 >> lc, ms, kHi);
    const uint64_t few = kHi ? 0 : objective_few(lc);  // (both bounds take one lane a box there)
    if (a.pinfo != nullptr && lc > 0 && a.max_boxes > few && a.chain.pure_objective &&
        fsmem + 1024 <= (size_t)max_dynamic_smem()) {
      auto siblings = chain_siblings_kernel<kMode, kHi>;
      // a block a tile while they are resident at once, else a warp a tile
      const uint64_t tiles = (a.max_boxes + 31) / 32, most = 512 * 32 / kObjThreads;
      uint64_t grid = resident_blocks(std::max(tiles, most), siblings, kObjThreads, fsmem);
      if (grid < tiles) grid = std::min(grid, std::max((tiles + 3) / 4, most));
      siblings<<<(unsigned)grid, kObjThreads, fsmem, s>>>(a, chains > 0 ? 1 : 0, 32 >> lc, (int)few);
      return cudaGetLastError();
    }
  }
  // few boxes of a program that is not tiny: lane groups for both bounds, in a
  // kernel of its own (their registers cost 9 % at 50,001 boxes).  Host boxes,
  // n = 64: 300 boxes 750 -> 190 us, 12,000 boxes 1,003 -> 849; 30,000 and 60,000
  // as one lane a box; n = 4, 30 instructions: 3,000 boxes 87 us by one lane, 91
  // by groups.
  auto kernel = chain_objective_kernel<kMode, kFused, kHi>;
  if constexpr (kHi && kMode == 0)
    if (a.max_boxes <= 16384 && a.prog_len > 64) kernel = chain_objective_kernel<kMode, kFused, kHi, true>;
  const size_t smem = objective_smem(a);
  const uint64_t grid = resident_blocks((a.max_boxes * 32 + kObjThreads - 1) / kObjThreads, kernel, kObjThreads, smem);
  kernel<<<(unsigned)grid, kObjThreads, smem, s>>>(a, chains > 0 ? 1 : 0);
  return cudaGetLastError();
}

// The role's one launch: regions of one box whose results go straight to the
// host (EvalArgs::flags is then free for the objective's blocks).  8,192 at
// most: with 16,384 the constraints fill the GPU by themselves, with their own
// kernel's eight warps a tile (n = 64: 226 us in two launches, 255 in one).
constexpr uint64_t kRoleMost = 8192;
// Above this many of them the objective's values are shared (512 regions, n =
// 32: 116 us by lane groups, 90 us for 1,024 shared).
constexpr uint64_t kRoleFew = 256;
static bool role_fits(const EvalArgs& a)
{
  return a.max_boxes <= kRoleMost && a.flags != nullptr && a.out_ub == nullptr && a.pinfo != nullptr && a.log2C < 0 && a.chain.pure_objective &&
         a.chain.n_seg > 1 &&
         (kObjThreads / 32) * family_bytes(1, a.max_slots, false) + 1024 <= (size_t)max_dynamic_smem();
}

static cudaError_t launch_role(const EvalArgs& a, cudaStream_t s)
{
  const bool share = a.max_boxes > kRoleFew;
  int lb = 5;
  while (lb > 0 && (a.max_boxes >> lb) < (uint64_t)sm_count() * 2) --lb;
  const uint64_t most = (uint64_t)sm_count() * 4;
  const uint64_t tiles = (a.max_boxes + 31) / 32, groups = (a.max_boxes * 32 + kObjThreads - 1) / kObjThreads;
  const uint64_t objective = share ? tiles : std::min(groups, most);
  const uint64_t constraints = std::min<uint64_t>((a.max_boxes + (1ull << lb) - 1) >> lb, most);
  const size_t smem = std::max(tile_smem_bytes(a.n_vars, a.max_slots, 1 << lb),
                               share ? (kObjThreads / 32) * family_bytes(1, a.max_slots, false) : objective_smem(a));
  EvalArgs ca = a, oa = a;
  ca.flags = nullptr;
  oa.out_flag = a.flags;
  oa.flags = nullptr;
  chain_role_kernel<<<(unsigned)(objective + constraints), kObjThreads, smem, s>>>(ca, oa, lb, (unsigned)objective,
                                                                                   share ? 1 : 0);
  return cudaGetLastError();
}

bool chain_fits(const EvalArgs& a)
{
  // the statics of the kernel take under 1 KiB beside the tile
  return a.chain.n_seg > 0 &&
         tile_smem_bytes(a.n_vars, a.pinfo != nullptr ? a.max_slots : 0, 32) + 1024 <= (size_t)max_dynamic_smem();
}

// Whether the passes here beat the interpreter's one launch.  They save three
// quarters of the <= chains' time, for a second launch and the staging of every
// box, worth about 3/4 of a term a variable (more where many boxes meet tiles so
// large that fewer than 16 warps of them fit an SM) and 3/2 a chain; `saved` is
// what is left, in quarters of a term a box.  Boxes, both bounds, interpreter against
// here: n = 4, one constraint (30 instructions), 20,000 boxes 26 and 39 us,
// 65,536 boxes 49 and 47, 524,288 boxes 220 and 148; n = 8, three constraints
// (145), 2,000 boxes 56 and 46, 131,072 boxes 359 and 126; n = 2, one
// constraint (6), 524,288 boxes 32 and 44; n = 200, one linear constraint, 4 warps,
// 20,000 boxes 177 and 335.  Few boxes of a long program: here
// lane groups form the objective faster (64 terms, 300 boxes 48 and 19 us).
// Chains with other readers keep the interpreter's arithmetic here, a warp
// each, so they need many boxes, and <= chains beside them to pay: sixteen ==
// chains of n = 24, 1,000 boxes 291 and 760 us; two chains of n = 24, one ==,
// 8,192 boxes 247 and 316, 131,072 boxes 1,427 and 986.
static bool general_pays(const EvalArgs& a, int mode, int64_t boxes, int64_t saved)
{
  const ChainTab& t = a.chain;
  const bool pure = t.pure_objective != 0;
  // the solver's children and parents: with many of them the chains fill the
  // GPU (256 parents x 4 children, sixteen == chains, n = 24: 8.6 and 10.8 ms)
  if (mode == 1 || mode == 3 || mode == 6) return boxes >= 8192 || (pure && t.general <= 4);
  // a role's one launch (n = 12, 1,024 regions, four == chains 134 and 103 us,
  // eight 146 and 168)
  if (mode == 0 && role_fits(a)) return t.general <= 4;
  const int64_t terms = t.general_terms;
  // few boxes: the objective by lane groups, or most of the chains <= ones
  // (n = 24, two constraints, one ==, 300 boxes 223 and 191 us; twelve, two ==,
  // 1,024 regions of an aggregate 433 and 337)
  if (pure && a.prog_len >= 200 && boxes < 8192)
    return mode == 4 ? 2 * t.constraint_terms >= 5 * terms : boxes <= 512 && t.general <= 2;
  if (boxes < 8192) return false;
  if (t.constraint_terms >= 2 * terms && saved >= 160 && saved * boxes >= 12000000) return true;
  if (!pure) return false;
  // 180 boxes a term of an average such chain keep the other warps busy, 80
  // regions, whose variables come from the cache (n = 24, two constraints, one
  // ==, 16,384 regions 434 and 327 us, 16,384 boxes 314 and 370)
  if (2 * t.constraint_terms >= terms && saved * boxes >= 2000000 && boxes >= 16384 &&
      boxes * t.general >= (a.pinfo != nullptr ? 80 : 180) * terms)
    return true;
  // between one wave and many, several chains spread over the warps (n = 12,
  // four == chains, 16,384 boxes 178 and 132 us; 524,288 boxes 2,014 and 2,030)
  return (t.general >= 2 && a.prog_len >= 140 && boxes >= 32768 && boxes <= 262144) ||
         (t.general >= 4 && a.prog_len >= 86 && boxes >= 16384 && boxes < 98304);
}

bool chain_pays(const EvalArgs& a, int mode)
{
  const ChainTab& t = a.chain;
  const int64_t boxes = (int64_t)a.max_boxes, len = a.prog_len;
  const int64_t tiles = max_dynamic_smem() / (int64_t)(tile_smem_bytes(a.n_vars, a.pinfo ? a.max_slots : 0, 32) + 1024);
  const int64_t warps = tiles * std::max(1, std::min(t.constraints + t.general, kTileWarps));
  // (regions read one parent's variables, from the cache)
  const bool waits = boxes > 32 * tiles * sm_count() && warps < (a.pinfo != nullptr ? 6 : 16);
  const int64_t saved = 4ll * t.constraint_terms - (waits ? 48ll * a.n_vars / warps : 3ll * a.n_vars) - 6ll * t.constraints;
  if (t.general > 0) return general_pays(a, mode, boxes, saved);
  if (mode == 1 || mode == 3 || mode == 6) return true;  // in the solver no form or size lost
  const bool region = a.pinfo != nullptr, both = mode == 4 || a.out_ub != nullptr;
  if (t.constraints == 0) {
    // the objective alone: the same work on either side, the program staged
    // there, lane groups or half the bounds here
    if (mode == 4) return len >= 45 || (len >= 15 && boxes <= 8);
    if (region) return true;
    if (both) return (len > 64 && boxes <= 10240) || (len >= 5 && boxes >= 98304);
    return len >= 12 || (len > 3 && boxes >= 65536);
  }
  const bool warped = t.constraints >= 2;  // a tile has a warp a chain
  if (mode == 4)  // n = 4, 30 instructions: 16,384 regions 50 and 65 us, 65,536 74 and 66
    return len >= 20 && ((len >= 72 && !waits) || saved * boxes >= (warped ? 2500000 : 3200000)) &&
           (len >= 40 || 2 * t.constraint_terms >= len);
  // n = 8, two constraints, 60 instructions, 32,768 regions 98 and 64 us; n = 4,
  // one, 30 instructions 49 and 63
  if (region)
    return role_fits(a) || (len >= 64 && !waits) || saved * boxes >= (warped && boxes >= 24576 ? 600000 : 1600000);
  // the second launch weighs less the longer the first is
  const int64_t need = boxes >= 90000                                    ? 1600000
                       : boxes >= 50000 || (boxes >= 28000 && warped) ? 2000000
                                                                         : 4200000;
  if (both)
    return saved * boxes >= need || (boxes <= 16384 && len >= 72 + boxes / 140 && (saved >= 64 || boxes <= 2048));
  return (len >= 64 && !waits) || saved * boxes >= need * 7 / 10 || (len >= 30 && boxes <= 512);
}

cudaError_t launch_chain(const EvalArgs& a, int mode, cudaStream_t s)
{
  if (mode == 0 && role_fits(a)) return launch_role(a, s);
  if (mode == 0) return a.out_ub != nullptr ? launch_chain_t<0, false, true>(a, s) : launch_chain_t<0, false, false>(a, s);
  if (mode == 6) return launch_chain_t<0, true, false>(a, s);
  if (mode == 1) return launch_chain_t<1, false, false>(a, s);
  if (mode == 4) return launch_chain_t<4, false, true>(a, s);
  return launch_chain_t<3, false, false>(a, s);
}

template <int kMode, bool kFused, bool kHi>
static cudaError_t allow_both(int max_smem)
{
  cudaError_t e = allow_dynamic_smem(chain_constraints_kernel<kMode, kFused>, max_smem);
  if constexpr (!kFused && kMode != 3)
    if (e == cudaSuccess) e = allow_dynamic_smem(chain_siblings_kernel<kMode, kHi>, max_smem);
  if constexpr (kHi && kMode == 0)
    if (e == cudaSuccess) e = allow_dynamic_smem(chain_objective_kernel<kMode, kFused, kHi, true>, max_smem);
  return e == cudaSuccess ? allow_dynamic_smem(chain_objective_kernel<kMode, kFused, kHi>, max_smem) : e;
}

cudaError_t set_chain_kernel_attributes(int max_smem)
{
  cudaError_t e = allow_dynamic_smem(chain_role_kernel, max_smem);
  if (e == cudaSuccess) e = allow_both<0, false, true>(max_smem);
  if (e == cudaSuccess) e = allow_both<0, false, false>(max_smem);
  if (e == cudaSuccess) e = allow_both<0, true, false>(max_smem);
  if (e == cudaSuccess) e = allow_both<1, false, false>(max_smem);
  if (e == cudaSuccess) e = allow_both<4, false, true>(max_smem);
  if (e == cudaSuccess) e = allow_both<3, false, false>(max_smem);
  return e;
}

}  // namespace cmn
